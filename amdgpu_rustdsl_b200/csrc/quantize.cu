// Device quantisers that produce the path's inputs from bf16 activations: the step in front of the attention kernels.
//
// The reference has no device code for this (its only FMHA quantiser is host code in the test harness, tests/gpu/ref_host.cpp:239-254;
// its device quantiser `quant_mxfp8_bf16_k` serves GEMM operands with 1x128 blocks and another scale rule,
// crates/amdgpu-kernels/src/rows/mxquant.rs:9-11,153). The rule restated here is the harness's:
//   Q, K: per 32 elements of the head dim  E8M0 = clamp(floor(log2 amax) - 8 + 127, 0, 254), elements e4m3(x * 2^-(E8M0 - 127)) rounded
//         to nearest even, saturating at 448; Q is multiplied by log2(e) / sqrt(128) first (`mul`), K by 1;
//   V:    per tensor  descale = amax / 448, elements e4m3(x / descale).
// All arithmetic is f32 with one rounding per operation, in the order written, so that the CPU restatement in the test oracle matches
// bit for bit. Inputs must be finite. Both kernels are pure streaming: 2 bytes in, 1 (+ 1/32) byte out per element.
#include "kernels.h"

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <type_traits>

namespace b200mx {

namespace {

__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
    uint16_t h;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(h) : "f"(hi), "f"(lo));
    return h;
}

// Programmatic dependent launch, both sides: the launch behind this one may be scheduled while this grid runs, and above the wait nothing reads or writes
// global memory: there are only the hints below. A short prompt's chain (Q, K, V, attention) is launches more than work.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Asks L2 for the line at `p`, one thread per 128 bytes of a warp's 16-byte vectors (all lines of them where x is 128-byte aligned, all but the last elsewhere). Allowed
// in front of the wait: nothing is read, and L2 is where a write of the grid before would land too. A grid's first vectors then come from DRAM while the last blocks of the
// grid before still run. Launches in a graph, without and with it: Q, K and V of B1 H8 HK2 S1000 6.6 and 6.0 us, B1 H16 HK4 S2048 11.1 and 10.5; Q or K of 1.2 M vectors 6.8
// and 6.3, of 16.8 M 66.8 and 66.1; V of 2.1 M 17.1 and 16.8, of 16.8 M 113.5 and 111.2.
__device__ __forceinline__ void prefetch_vec(const uint4* p) {
    if ((threadIdx.x & 7u) == 0u) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// A 16-byte read-once load. Volatile, so that it stays behind the wait above, and not of the non-coherent kind, which is for data that nothing writes while
// the grid runs.
__device__ __forceinline__ uint4 ld_vec(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// 8 consecutive elements (16 bytes in, 8 bytes out) of one 32-element block per lane; 4 lanes = one block, 16 lanes = one row of 128. All 32 lanes
// take part (shuffles); a lane that is not live has zeros and stores nothing.
__device__ __forceinline__ void quantize_qk_vec(const uint4 raw, bool live, float mul, unsigned lane, unsigned long long t, uint2* __restrict__ out, uint32_t* __restrict__ scales) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    float y[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        y[2 * i] = __fmul_rn(__uint_as_float(w[i] << 16), mul);
        y[2 * i + 1] = __fmul_rn(__uint_as_float(w[i] & 0xFFFF0000u), mul);
    }
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(y[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    // floor(log2 amax) of a normal f32 is its exponent field - 127; zero and subnormal maxima end at the lower clamp either way
    int eb = static_cast<int>((__float_as_uint(amax) >> 23) & 0xFFu) - 8;
    eb = eb < 0 ? 0 : (eb > 254 ? 254 : eb);
    // x * 2^(127 - eb) as two exact multiplications by normal powers of two (the exponent 127 - eb lies in [-127, 127]; a value that
    // an intermediate product flushes or rounds is far below the smallest e4m3 step in the end and encodes as zero either way)
    const int sh = 127 - eb, sh1 = sh >> 1, sh2 = sh - sh1;
    const float s1 = __uint_as_float(static_cast<uint32_t>(127 + sh1) << 23), s2 = __uint_as_float(static_cast<uint32_t>(127 + sh2) << 23);
    uint32_t b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        b[i] = e4m3x2(__fmul_rn(__fmul_rn(y[4 * i], s1), s2), __fmul_rn(__fmul_rn(y[4 * i + 1], s1), s2)) |
               (e4m3x2(__fmul_rn(__fmul_rn(y[4 * i + 2], s1), s2), __fmul_rn(__fmul_rn(y[4 * i + 3], s1), s2)) << 16);
    }
    if (live) out[t] = make_uint2(b[0], b[1]);
    // the row's four scale bytes: lanes 0, 4, 8, 12 of each 16-lane half hold them
    const uint32_t e1 = __shfl_down_sync(0xFFFFFFFFu, static_cast<uint32_t>(eb), 4);
    const uint32_t e2 = __shfl_down_sync(0xFFFFFFFFu, static_cast<uint32_t>(eb), 8);
    const uint32_t e3 = __shfl_down_sync(0xFFFFFFFFu, static_cast<uint32_t>(eb), 12);
    if (live && (lane & 15u) == 0u) scales[t >> 4] = static_cast<uint32_t>(eb) | (e1 << 8) | (e2 << 16) | (e3 << 24);
}

// kVecs 16-byte loads of a thread are in flight before the first is used: bound by DRAM, and one load per thread at a time does not cover its latency.
template <int kVecs>
__global__ void __launch_bounds__(256) quantize_qk_kernel(const uint4* __restrict__ x, unsigned long long rows, float mul,
                                                          uint2* __restrict__ out, uint32_t* __restrict__ scales) {
    pdl_launch();
    const unsigned long long n_threads = rows * 16ull, step = static_cast<unsigned long long>(gridDim.x) * (256u * kVecs);
    const unsigned lane = threadIdx.x & 31u;
    // the warp's first vector; whole warps stay in the loop together: the shuffles need all lanes
    const unsigned long long first = static_cast<unsigned long long>(blockIdx.x) * (256u * kVecs) + (threadIdx.x & ~31u);
    // Behind a branch in the wide form: without it the kernel compiles to 40 registers, not 46, and is slower for it (Q or K of 16.8 M vectors 76.8 us, so 71.5, both with
    // a grid of 8 CTAs per SM)
    if (kVecs == 1 || first < n_threads) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            if (first + lane + 256u * i < n_threads) prefetch_vec(x + first + lane + 256u * i);
        }
    }
    pdl_wait();
    for (unsigned long long t0 = first; t0 < n_threads; t0 += step) {
        uint4 raw[kVecs];
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            const unsigned long long t = t0 + lane + 256u * i;
            raw[i] = t < n_threads ? ld_vec(x + t) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
            const unsigned long long t = t0 + lane + 256u * i;
            quantize_qk_vec(raw[i], t < n_threads, mul, lane, t, out, scales);
        }
    }
}

__device__ __forceinline__ float amax_vec(float amax, const uint4 raw) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w[i] << 16)), fabsf(__uint_as_float(w[i] & 0xFFFF0000u))));
    return amax;
}

__device__ __forceinline__ float amax_warp(float amax) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    return amax;
}

__device__ __forceinline__ float v_descale_of(float amax) { return amax > 0.0f ? __fdiv_rn(amax, 448.0f) : 1.0f; }

// x / vd rounded to nearest even, from r = 1 / vd rounded to nearest: q = x r is within an ulp, and one residual correction rounds it
// correctly (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, 1990, theorem 7.2). vd is in
// [kDivLo, kDivHi]: no residual that matters underflows (|x| <= 448 vd (1 + 2^-23); a quotient under 2^-11 is the byte 0 either way). A division
// costs a tenth of these three instructions' rate and was what the kernel waited for.
__device__ __forceinline__ float div_by(float x, float vd, float r) {
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(-__fmaf_rn(q, vd, -x), r, q);   // the residual with its sign turned: x = -0 then stays -0 (the other way round it ends as -0 + 0)
}
constexpr float kDivLo = 0x1p-90f, kDivHi = 0x1p100f;

template <bool kFast>
__device__ __forceinline__ uint2 quantize_v_vec(const uint4 raw, float vd, float r) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    auto q = [&](uint32_t bits) { return kFast ? div_by(__uint_as_float(bits), vd, r) : __fdiv_rn(__uint_as_float(bits), vd); };
    uint32_t b[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        b[i] = e4m3x2(q(w[2 * i] << 16), q(w[2 * i] & 0xFFFF0000u)) | (e4m3x2(q(w[2 * i + 1] << 16), q(w[2 * i + 1] & 0xFFFF0000u)) << 16);
    }
    return make_uint2(b[0], b[1]);
}

// descale = {0, 0} in front of the running maximum. A kernel of the chain and not a memset, around which no grid starts early: in a graph, Q, K and V of B1 H16 HK4 S2048
// 14.4 us with the memset and 11.1 with this, B2 H32 HK8 S3000 33.5 and 29.6 (both without the hints above). It costs the host 0.8 us more a call, which is what a caller
// sees whose GPU has nothing else to do: V of 2304 rows again and again 8.0 and 8.8 us.
__global__ void clear_descale_kernel(float* descale) {
    pdl_launch();
    pdl_wait();
    if (threadIdx.x < 2u) descale[threadIdx.x] = 0.0f;
}

template <int kVecs>
__global__ void __launch_bounds__(256) amax_kernel(const uint4* __restrict__ x, unsigned long long n_vec, uint32_t* __restrict__ amax_bits) {
    float amax = 0.0f;
    const unsigned long long step = static_cast<unsigned long long>(gridDim.x) * (256u * kVecs), first = static_cast<unsigned long long>(blockIdx.x) * (256u * kVecs) + threadIdx.x;
    pdl_launch();
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
        if (first + 256u * i < n_vec) prefetch_vec(x + first + 256u * i);
    }
    pdl_wait();
    for (unsigned long long t0 = first; t0 < n_vec; t0 += step) {
        uint4 raw[kVecs];
#pragma unroll
        for (int i = 0; i < kVecs; ++i) raw[i] = t0 + 256u * i < n_vec ? ld_vec(x + t0 + 256u * i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < kVecs; ++i) amax = amax_vec(amax, raw[i]);
    }
    amax = amax_warp(amax);
    __shared__ float part[8];
    if ((threadIdx.x & 31u) == 0u) part[threadIdx.x >> 5] = amax;
    __syncthreads();
    if (threadIdx.x == 0u) {
#pragma unroll
        for (int i = 1; i < 8; ++i) amax = fmaxf(amax, part[i]);
        atomicMax(amax_bits, __float_as_uint(amax));   // non-negative floats order like their bit patterns
    }
}

// Walks the vectors from the last to the first: the amax pass before it read them in rising order, so the last ones are still in L2.
template <int kVecs>
__global__ void __launch_bounds__(256) quantize_v_kernel(const uint4* __restrict__ x, unsigned long long n_vec, uint2* __restrict__ out,
                                                         float* __restrict__ descale) {
    pdl_launch();
    pdl_wait();
    const float amax = __uint_as_float(reinterpret_cast<const volatile uint32_t*>(descale)[1]);
    const float vd = v_descale_of(amax);
    if (blockIdx.x == 0 && threadIdx.x == 0) descale[0] = vd;
    const unsigned long long step = static_cast<unsigned long long>(gridDim.x) * (256u * kVecs);
    auto pass = [&](auto fast_c, float r) {
        constexpr bool kFast = decltype(fast_c)::value;
        for (unsigned long long t0 = static_cast<unsigned long long>(blockIdx.x) * (256u * kVecs) + threadIdx.x; t0 < n_vec; t0 += step) {
            uint4 raw[kVecs];
#pragma unroll
            for (int i = 0; i < kVecs; ++i) raw[i] = t0 + 256u * i < n_vec ? ld_vec(x + (n_vec - 1u - t0 - 256u * i)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int i = 0; i < kVecs; ++i) {
                const uint2 b = quantize_v_vec<kFast>(raw[i], vd, r);
                if (t0 + 256u * i < n_vec) out[n_vec - 1u - t0 - 256u * i] = b;
            }
        }
    };
    if (vd >= kDivLo && vd <= kDivHi) pass(std::true_type{}, __frcp_rn(vd));
    else pass(std::false_type{}, 0.0f);
}

// A small V in one launch: a cluster of 8 CTAs keeps it in registers between the maximum, exchanged through distributed shared memory, and the
// quantisation. The general form is three launches (clear, maximum, quantise) and reads V twice.
constexpr unsigned kSmallCtas = 8, kSmallThreads = 1024, kSmallVecs = 4, kSmallMax = kSmallCtas * kSmallThreads * kSmallVecs;
__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallThreads)
quantize_v_small_kernel(const uint4* __restrict__ x, unsigned n_vec, uint2* __restrict__ out, float* __restrict__ descale) {
    namespace cg = cooperative_groups;
    // A CTA's shared memory may only be written by another one once it is known to have started: every thread arrives here and waits in front of the
    // exchange, behind the loads. (Being scheduled as one cluster does not give that order, nor does the wait for the grid before.)
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    pdl_launch();
    __shared__ float part[kSmallThreads / 32];
    __shared__ float cta_amax[kSmallCtas];   // [source CTA], written by all of them
    const cg::cluster_group cluster = cg::this_cluster();
    const unsigned tid = blockIdx.x * kSmallThreads + threadIdx.x;
    uint4 raw[kSmallVecs];
#pragma unroll
    for (unsigned i = 0; i < kSmallVecs; ++i) {
        const unsigned t = tid + i * (kSmallCtas * kSmallThreads);
        if (t < n_vec) prefetch_vec(x + t);
    }
    pdl_wait();
#pragma unroll
    for (unsigned i = 0; i < kSmallVecs; ++i) {
        const unsigned t = tid + i * (kSmallCtas * kSmallThreads);
        raw[i] = t < n_vec ? ld_vec(x + t) : make_uint4(0u, 0u, 0u, 0u);
    }
    float amax = 0.0f;
#pragma unroll
    for (unsigned i = 0; i < kSmallVecs; ++i) amax = amax_vec(amax, raw[i]);
    amax = amax_warp(amax);
    if ((threadIdx.x & 31u) == 0u) part[threadIdx.x >> 5] = amax;
    __syncthreads();
    asm volatile("barrier.cluster.wait;" ::: "memory");
    if (threadIdx.x < 32u) {
        amax = amax_warp(part[threadIdx.x]);
        if (threadIdx.x < kSmallCtas) *cluster.map_shared_rank(&cta_amax[blockIdx.x], threadIdx.x) = amax;
    }
    cluster.sync();   // (nobody touches another CTA's shared memory behind it)
    amax = cta_amax[0];
#pragma unroll
    for (unsigned i = 1; i < kSmallCtas; ++i) amax = fmaxf(amax, cta_amax[i]);
    const float vd = v_descale_of(amax);
    if (tid == 0u) {
        descale[0] = vd;
        reinterpret_cast<uint32_t*>(descale)[1] = __float_as_uint(amax);   // what the general form leaves there
    }
    const bool fast = vd >= kDivLo && vd <= kDivHi;
    const float r = fast ? __frcp_rn(vd) : 0.0f;
#pragma unroll
    for (unsigned i = 0; i < kSmallVecs; ++i) {
        const unsigned t = tid + i * (kSmallCtas * kSmallThreads);
        if (t < n_vec) out[t] = fast ? quantize_v_vec<true>(raw[i], vd, r) : quantize_v_vec<false>(raw[i], vd, r);
    }
}

// Blocks of 256 threads with `vecs` vectors each; grid-stride beyond `per_sm` CTAs per SM
int grid_for(unsigned long long n_vec, unsigned vecs, unsigned per_sm = 8u) {
    const unsigned long long blocks = (n_vec + 256u * vecs - 1) / (256u * vecs), cap = 1ull * per_sm * static_cast<unsigned long long>(current_sm_count());
    return static_cast<int>(blocks < cap ? (blocks ? blocks : 1) : cap);
}

template <typename... Params, typename... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), unsigned grid, unsigned threads, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// From 4 vectors per thread of a full machine on: the wide form then still has every SM's thread slots filled.
constexpr unsigned long long kWideVecs = 4ull * 148ull * 2048ull;

}  // namespace

cudaError_t launch_quantize_qk(const void* x_bf16, unsigned long long rows, float mul, void* out_e4m3, void* out_scales, cudaStream_t stream) {
    const unsigned long long n_vec = rows * 16ull;
    const bool wide = n_vec >= kWideVecs;
    // An SM holds 5 CTAs of the wide form (46 registers): 10 are two whole rounds of them. With 8, whose second round is three fifths of one, 2.1 M vectors took 10.1 us, so
    // 9.2 (1.6 M: 7.7 and 8.0; 4.2 M: 18.4 and 17.3; 16.8 M: 72.1 and 66.1)
    return launch_pdl(wide ? quantize_qk_kernel<4> : quantize_qk_kernel<1>, grid_for(n_vec, wide ? 4u : 1u, wide ? 10u : 8u), 256u, stream, static_cast<const uint4*>(x_bf16), rows, mul,
                      static_cast<uint2*>(out_e4m3), static_cast<uint32_t*>(out_scales));
}

cudaError_t launch_quantize_v(const void* x_bf16, unsigned long long n_elems, void* out_e4m3, float* descale, cudaStream_t stream) {
    const unsigned long long n_vec = n_elems / 8;
    const uint4* x = static_cast<const uint4*>(x_bf16);
    uint2* out = static_cast<uint2*>(out_e4m3);
    if (n_vec <= kSmallMax) return launch_pdl(quantize_v_small_kernel, kSmallCtas, kSmallThreads, stream, x, static_cast<unsigned>(n_vec), out, descale);
    cudaError_t e = launch_pdl(clear_descale_kernel, 1u, 32u, stream, descale);   // [0] the descale, [1] the running maximum's bits
    if (e != cudaSuccess) return e;
    const bool wide = n_vec >= kWideVecs;
    const unsigned grid = grid_for(n_vec, wide ? 4u : 1u);
    e = launch_pdl(wide ? amax_kernel<4> : amax_kernel<1>, grid, 256u, stream, x, n_vec, reinterpret_cast<uint32_t*>(descale) + 1);
    if (e != cudaSuccess) return e;
    return launch_pdl(wide ? quantize_v_kernel<4> : quantize_v_kernel<1>, grid, 256u, stream, x, n_vec, out, descale);
}

}  // namespace b200mx
