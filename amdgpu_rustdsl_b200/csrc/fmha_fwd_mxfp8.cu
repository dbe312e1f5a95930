// MXFP8 attention forward, head dim 128, for sm_100a: the bodies of fmha_fwd_hd128_mxfp8_v3_{vs128, t128, kvsplit}.
//
// What one CTA computes (reference: crates/amdgpu-stage/src/attention/attn3.rs:260-755, block3.rs:79-356): for 128 query rows of
// one (batch, head) and a key range [key_lo, key_hi), out = softmax2(q k^T) v with
//   q k^T  : e4m3 x e4m3 with one E8M0 scale per 32 elements of the head dim on both sides (block-scaled tensor-core MMA),
//   softmax: base 2, no extra scale (the host folds log2(e)/sqrt(128) into Q before quantisation, tests/gpu/ref_host.cpp:238),
//            online over the keys with a lazily moved reference: the reference only moves when a row maximum passes it by
//            more than a threshold (crates/amdgpu-tile/src/softmax.rs:179-243; there O and the row sum are then rescaled, here P carries the
//            difference as its block scale);
//            sequences under 4 tiles move the reference on every tile (crates/amdgpu-stage/src/attention/state.rs:73-77),
//   P      : requantised to e4m3 (long sequences: with one E8M0 per row and 32 keys) before P V, and the row sum adds the *quantised* P (crates/amdgpu-tile/src/reduce.rs:163-173),
//   out    : O * v_descale / l as bf16 (state.rs:79-82), or for the split kernel the normalised f32 partial plus a base-2
//            log-sum-exp per row (block3.rs:291-356).
//
// Mapping onto the SM (not a translation of the gfx950 wave layout): a persistent kernel, one CTA of 16 warps per SM, each CTA walking
// work items (128 query rows of one (batch, head[, split])) with its rings, buffers and barriers running on across items.
// The four service warps run their loops with all 32 lanes in step on warp-uniform values and let an elected lane issue the tcgen05 /
// TMA instructions (operands then stay in uniform registers).
//   warp  0    Q K^T issuer: S[g % 2] = Q K_g^T as kind::mxf8f6f4.block_scale tcgen05.mma, both operands in swizzled shared memory,
//              the E8M0 factors copied to TMEM with tcgen05.cp. Two score tiles are always ahead of the softmax.
//   warp  1    Q / K producer: TMA loads of the Q tile (double buffered across items) and of the K ring, plus the 4-byte-per-row scale
//              bytes of both, which a TMA box cannot express: 4-byte asynchronous copies straight into the 32x16-byte layout tcgen05.cp
//              expects, arriving on the tile's barrier. In the set-up it initialises all barriers and sends out the first Q, K and V tiles.
//   warp  2    P V issuer: O += P_g V_g with P from TMEM and V (keys x head dim, i.e. MN-major B) from shared memory. The B operand
//              is 144 wide: 128 head dims plus 16 columns of a tile of e4m3 ones, so that O[:, 128..143] (= the L columns) holds the
//              row sums of the *quantised* P at no ALU cost (the reference sums P with a matrix instruction too, reduce.rs:163-173).
//              It has a thread of its own: the tensor pipe takes MMAs from one thread at its full rate, but a thread that shares its
//              scheduler with softmax warps only gets an instruction in every few clocks.
//   warp  3    V producer: TMA loads of the V ring (K is freed after Q K^T, V after P V, so the two rings run apart).
//   warps 4-11 softmax, two warpgroups: warpgroup p works on the tiles with counter g = p (mod 2). Thread r of a group owns query row
//              r = TMEM lane r: it reads the row's 128 scores from tensor memory and hands the S buffer back at once, converts block by
//              block of 32 keys with the block's own reference, writes P (packed e4m3) with tcgen05.st and, when they change, the
//              row's block scales to shared memory. The references travel between the groups through 8-byte shared-memory slots
//              {value, tile counter}, off the critical path.
//   warps 12-15 epilogue, one warpgroup: takes an item's O and row sums out of tensor memory when its last P V is done, hands the
//              columns back (the next item's first P V waits for that), normalises, stages the tile in shared memory and stores it
//              with TMA (bf16 output, or the split kernel's partial), while the softmax warpgroups are on the next item's tiles.
//              Merges the two halves of an item cut between a pair of CTAs; in the fused instantiations merges a row block's partials.
//   Every thread starts with 128 registers; the service warps then keep 56, the softmax warps take 176 and the epilogue warps 104
//   (setmaxnreg: the roles' shares must come out of the CTA's launch allocation).
// TMEM columns: S0 [0,128) S1 [128,256) O [256,384) L [384,400) P0 [400,432) P1 [432,464) SFQ [464,468) SFK0 [468,472) SFK1 [472,476)
// SFP [476,480) SFV [480,488).
#include "kernels.h"
#include "ptx_sm100.cuh"

#include <cuda_bf16.h>

#include <atomic>
#include <mutex>
#include <type_traits>
#include <cuda_fp8.h>

namespace b200mx {
using namespace sm100;

namespace {

constexpr int kRows = 128;          // query rows per CTA tile
constexpr int kKeys = kKeysPerTile; // keys per tile (128)
constexpr int kStages = 4;          // depth of the K ring and of the V ring (freed separately: K after Q K^T, V after P V)
// The four service warps get the lowest warp ids, one per scheduler (scheduler = warp % 4). Softmax = warps 4-19: a warp's TMEM lane
// quadrant is warp % 4, so any four consecutive warps cover the 128 rows.
constexpr int kMmaWarp = 0, kKProducerWarp = 1, kPvWarp = 2, kVProducerWarp = 3, kFirstSoftmaxWarp = 4, kFirstEpilogueWarp = 12;
// A softmax thread owns a whole score row of a tile: 128 scores in registers, read from tensor memory once. 4 service + 8 softmax + 4
// epilogue warps: every scheduler has one service, two softmax and one epilogue warp and 16 K registers to deal out among them.
constexpr int kCols = 128;                  // score columns per softmax thread
constexpr int kThreads = 32 * (4 + 8 + 4);   // 4 service warps, 8 softmax warps, 4 epilogue warps
// The register file (64 K registers) is dealt out unevenly once the roles part: every thread starts with kMaxRegs, the service and the
// epilogue warpgroups give most of theirs back and the two softmax warpgroups take them.
#ifndef MXA_SERVICE_REGS
#define MXA_SERVICE_REGS 56
#define MXA_SOFTMAX_REGS 176
#define MXA_EPILOGUE_REGS 104
#endif
constexpr int kMaxRegs = 128;
constexpr int kServiceRegs = MXA_SERVICE_REGS, kSoftmaxRegs = MXA_SOFTMAX_REGS, kEpilogueRegs = MXA_EPILOGUE_REGS;
// setmaxnreg.inc waits, without a bound, until the CTA's own pool has the registers, and the pool is what the CTA got at launch
// (kThreads x kMaxRegs), not the SM's register file: the roles together must never ask for more than that.
static_assert(kThreads * kMaxRegs <= 65536, "the CTA must fit the register file at launch");
static_assert(4 * kServiceRegs + 8 * kSoftmaxRegs + 4 * kEpilogueRegs <= (kThreads / 32) * kMaxRegs, "the roles' registers come out of the CTA's launch allocation");
static_assert(kServiceRegs % 8 == 0 && kSoftmaxRegs % 8 == 0 && kEpilogueRegs % 8 == 0 && kServiceRegs >= 24 && kEpilogueRegs >= 24 && kSoftmaxRegs <= 256, "register file split");
constexpr uint32_t kTileBytes = 128 * 128;   // one e4m3 tile
constexpr uint32_t kSfBytes = 512;           // 128 rows x 4 scale bytes

constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO = 256, kColL = 384, kColP0 = 400, kColP1 = 432, kColSfQ = 464, kColSfK0 = 468, kColSfK1 = 472,
                   kColSfP = 476, kColSfV = 480;   // V block scales (extension): P's constant factors [476,480), V's factors [480,484) + the ones columns' [484,488)
constexpr uint32_t kTmemCols = 512;

// P = 2^(s - ref + kPOffset): the row's reference maps to 2^kPOffset.
// Long sequences (>= 4 key tiles): the reference is an integer, ceil(block maximum), and is left alone while a block's maximum stays
// within kLazyThreshold binades above it, so P <= 2^(5 + 3.5) = 362 < 448 never saturates e4m3. Integer references differ by exact powers of
// two, so the same keys give the same P mantissas whatever the reference: a KV split and the unsplit kernel then differ only by f32
// summation order (and where P is subnormal).
// Short sequences move the reference to the tile's own maximum on every tile whose maximum is less than kFollowWindow binades
// below it (so every tile's largest P is exactly 2^kPOffset, which is what keeps the error on sharply peaked rows at the level of
// the reference's short-sequence recipe: thr 120/512 vs target 131/512, crates/amdgpu-tile/src/softmax.rs:26-30).
constexpr float kPOffset = 5.0f;
constexpr float kLazyThreshold = 3.5f;
constexpr float kFollowWindow = 11.0f;
// Long sequences: O and L are in units of the row's base and a tile's P carries 2^(reference - base) as its block scale, as far as this many binades
// above the base; a row that grows further gets a new base. With a scalar V descale O holds e4m3 values: the products stay far inside f32 for 2^(8.5 + 60) x
// 2^8.8 (the largest e4m3 V) x 2^20 keys. With V block scales O holds V as it is, which may be near the end of bf16 and f32 itself, so only 8 are
// taken from it there; a row of normal scores grows by 4 or 5 over its first 128 keys' maximum.
template <bool kVbs>
constexpr float kRebase = kVbs ? 8.0f : 60.0f;
// Long sequences: the reference before any key with a score above -inf has been seen. Finite, so that scores of -inf (a whole block or tile of masked keys)
// give P = 0 and not the NaN of -inf - -inf.
constexpr float kNoRef = -3.402823466e38f;
constexpr uint32_t kFlagCausal = 0x8u;   // FMHA_MXFP8_FLAG_CAUSAL: selects the kCausal instantiations
constexpr uint32_t kFlagF32Partials = 0x10u;   // FMHA_MXFP8_FLAG_F32_PARTIALS: the split kernel's partial rows are f32, not f16
constexpr uint32_t kFlagNoTailSplit = 0x20u;   // FMHA_MXFP8_FLAG_NO_TAIL_SPLIT: never cut the last round's items in two

struct SmemLayout {
    // all tile buffers are 1024-byte aligned (128-byte swizzle atom = 8 rows x 128 B)
    static constexpr uint32_t q = 0;
    static constexpr uint32_t k = q + 2 * kTileBytes;   // two Q tiles: the next item's is loaded while the current one is in use
    static constexpr uint32_t v = k + kStages * kTileBytes;
    // 32 keys x 128 B of e4m3 1.0 behind the V ring: a second MN-major atom of the P V B operand, of which the MMA uses 16 columns,
    // so that O[:, 128..143] accumulates the row sums of P
    static constexpr uint32_t ones = v + kStages * kTileBytes;
    // two 16 KB staging tiles (128 rows x 64 bf16, 128-byte swizzle) for the output's TMA stores, one per warpgroup
    static constexpr uint32_t ostage = ones + 4096;
    static constexpr uint32_t sfq = ostage + 2 * 16384;
    static constexpr uint32_t sfk = sfq + 2 * kSfBytes;
    // [tile counter % 8][row 128] x {reference bits, tile counter}. A group that publishes tile g + 6 has finished g + 4, so P V of g + 2 and
    // with it that of g + 1 is done, so the other group is past its tile g + 1 and has read slot g: six slots are enough
    static constexpr uint32_t sfv = sfk + kStages * kSfBytes;    // V block scales of a key tile (extension), same 32 x 16-byte pattern as the K scales
    static constexpr uint32_t sf_one = sfv + kStages * kSfBytes;  // 512 bytes of E8M0 1.0: the factors of P and of the ones columns
    static constexpr uint32_t xref = sf_one + kSfBytes;
    // [item ordinal % 4][row 128]: the row's reference after the item's last tile, for the epilogue warpgroup. Four slots and a write
    // behind the wait for this parity's previous P V: with one-tile items a softmax group is otherwise two items ahead of the epilogue
    static constexpr uint32_t xfin = xref + 8 * 128 * 8;
    static constexpr uint32_t xstat = xfin + 4 * 128 * 4;         // [row 128] x {row sum, reference} of the partner's half item (launches as pairs)
    static constexpr uint32_t xlse = xstat + 128 * 8;             // fused merge: [row 128][split 8] log-sum-exps of the block being merged
    static constexpr uint32_t sfp = xlse + 128 * 8 * 4;          // P block scales, one buffer per softmax group, same 32 x 16-byte pattern
    static constexpr uint32_t bars = sfp + 2 * kSfBytes;
    // barriers (8 bytes each): q_full[2], q_empty[2], k_full[kStages], k_empty[kStages], v_full[kStages], v_empty[kStages], s_full[2], s_free[2],
    // p_full[2], o_done[2], o_free, o_full, four unused, peer_rdy, peer_data
    static constexpr uint32_t n_bars = 4 + 4 * kStages + 16;
    static constexpr uint32_t tmem_slot = bars + 8 * n_bars;
    static constexpr uint32_t abort_flag = tmem_slot + 4;
    static constexpr uint32_t last_flag = abort_flag + 4;   // fused merge: "this CTA brought the row block's arrival count to `splits`"
    static constexpr uint32_t total = last_flag + 4;
};
constexpr uint32_t kSmemBytes = SmemLayout::total + 1024;   // + slack to align the base to 1024
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget of one CTA");

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

// Two floats -> two e4m3 bytes (round to nearest even, saturating), `a` in the low byte.
__device__ __forceinline__ uint32_t cvt_e4m3x2(float a, float b) {
    uint16_t h;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(h) : "f"(b), "f"(a));
    return static_cast<uint32_t>(h);
}

// Four scores -> one 32-bit word of four e4m3 P values, key order = byte order.
__device__ __forceinline__ uint32_t p_word(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, float sh) {
    const uint32_t lo = cvt_e4m3x2(ex2_approx(__uint_as_float(s0) + sh), ex2_approx(__uint_as_float(s1) + sh));
    const uint32_t hi = cvt_e4m3x2(ex2_approx(__uint_as_float(s2) + sh), ex2_approx(__uint_as_float(s3) + sh));
    return lo | (hi << 16);
}

// The long-sequence conversion: the exp2 unit delivers 16 results per clock per SM, a quarter of what the score tiles need at full
// tensor rate, so two of every four P values are produced on the FMA pipe instead, straight as e4m3 bit patterns:
// byte = rne(8 (x + 7)) with x = log2 P, i.e. exponent field = floor(x) + 7 and a mantissa that is linear in the fraction of x
// (the piecewise-linear exp2 the reference uses for all of P, crates/amdgpu-tile/src/reduce.rs:94-113, docs/vendor-spec.md:271-281).
// The rounding, the clamp at zero and the packing are one conversion: 8 (x + 7) 2^-24 is a subnormal f16 whose bit pattern is the byte, and
// cvt.relu takes everything below (-inf scores too) to 0. So two values cost one two-wide fma and one conversion, against two clamped fma, an
// addition and a permute for doing the rounding in f32; the additions in front of the exp2 of the other two are also done two at a time.
// The linear mantissa overestimates 2^frac by 3.97 % on average; kFastBias shifts x so that the two kinds of P values agree on
// average, otherwise mixing them in one row sum would bias the weights.
constexpr float kFastBias = 0.0562f;
// Two f32 additions in one instruction (sm_100 has two-wide f32 add / mul / fma on 64-bit register pairs): a += c, b += c.
__device__ __forceinline__ void add2(uint32_t& a, uint32_t& b, float c) {
    unsigned long long p, q;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(a), "r"(b));
    asm("mov.b64 %0, {%1, %1};" : "=l"(q) : "f"(c));
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(p) : "l"(p), "l"(q));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(p));
}
// a *= c, b *= c in one instruction
__device__ __forceinline__ void mul2(uint32_t& a, uint32_t& b, float c) {
    unsigned long long p, q;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(a), "r"(b));
    asm("mov.b64 %0, {%1, %1};" : "=l"(q) : "f"(c));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(p), "l"(q));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(p));
}
// a = a x + c, b = b x + c in one instruction
__device__ __forceinline__ void fma2(uint32_t& a, uint32_t& b, float x, float c) {
    unsigned long long p, q, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "r"(a), "r"(b));
    asm("mov.b64 %0, {%1, %1};" : "=l"(q) : "f"(x));
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(c));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(p), "l"(q), "l"(r));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(p));
}
// max(a, 0) in the low and max(b, 0) in the high half, as f16 (subnormals kept)
__device__ __forceinline__ uint32_t cvt_relu_f16x2(float a, float b) {
    uint32_t h;
    asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(b), "f"(a));
    return h;
}
__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.volatile.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint2 ld_shared_v2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}

// Time stamps of logical block (0,0,0) for the first 32 key tiles (the analogue of the reference's in-kernel stamp buffer,
// docs/stamps.md): [role 4: softmax group 0, 1, score MMAs, P V MMAs][tile 32][slot 8] 64-bit SM clock values behind the first 37120 words of the trace buffer.
constexpr int kStampBase = 37120;
template <bool kTrace>
__device__ __forceinline__ void stamp_t(float* trace, int role, int tile, int slot) {
    if (kTrace && trace != nullptr && tile < 32) reinterpret_cast<long long*>(trace + kStampBase)[(role * 32 + tile) * 8 + slot] = clock64();
}

// O columns [col, col + 64) of this thread's lane *= f
__device__ __forceinline__ void scale_tmem64(uint32_t taddr, float f) {
    uint32_t a[32], b[32];
    tmem_ld32(taddr, a);
    tmem_ld32(taddr + 32, b);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < 32; c += 2) mul2(a[c], a[c + 1], f);
    tmem_st32(taddr, a);
#pragma unroll
    for (int c = 0; c < 32; c += 2) mul2(b[c], b[c + 1], f);
    tmem_st32(taddr + 32, b);
}

// One unit of work of the persistent kernel: 128 query rows against the key range of one split. The rows are 128 of one (batch, head), or, with
// the heads of a KV head packed (AttnParams::pack_shift), 128 >> pack_shift sequence rows of each of the 1 << pack_shift heads that share it:
// TMEM lane r is then sequence row row0 + (r >> pack_shift) of head head + r % (1 << pack_shift).
struct Item {
    uint32_t row0, head, batch, split, kv_head, key_lo, key_hi;
    uint32_t half;   // pairs: 0: the item's whole key range; 1 / 2: its first / second half, to be merged with the other CTA of the cluster
    int n_tiles;
};

// How a launch deals the key range of an item out within a cluster: not at all, the last round's items between pairs, every item between all CTAs.
enum Cluster { kNoCluster = 0, kPairs = 1, kCutAll = 2 };

template <bool kSplit, bool kCausal, Cluster kCluster, bool kPack>
__device__ __forceinline__ Item decode_item(uint32_t w, const AttnParams& p) {
    const uint32_t ps = kPack ? p.pack_shift : 0u;
    // w = (z * H + head) * n_qtiles + q tile: neighbouring CTAs work on neighbouring row blocks of one head, whose K / V they share in L2
    Item it;
    it.half = 0;
    const uint32_t part = w & ((1u << p.cut_log2) - 1u);   // kCutAll: unit w is part `part` of item w >> cut_log2
    if (kCluster == kCutAll) w >>= p.cut_log2;
    if (kCluster == kPairs && w >= p.tail_base) {   // a unit of the cut last round: half (w - tail_base) % 2 of item tail_base + (w - tail_base) / 2
        it.half = 1u + ((w - p.tail_base) & 1u);
        w = p.tail_base + ((w - p.tail_base) >> 1);
    }
    uint32_t x = w % p.n_qtiles, yz = w / p.n_qtiles;
    constexpr bool causal = kCausal && !kSplit;
    if (causal) {
        // Items in the order of falling work (the row block's visible keys): rank = (n_qtiles - 1 - q tile) * (H * B) + (batch * H + head).
        // The CTAs walk the ranks in rounds of gridDim.x, odd rounds backwards, so that the CTA that got the heaviest item of one round
        // gets the lightest of the next and every CTA ends with about the same number of key tiles.
        const uint32_t round = w / gridDim.x, base = round * gridDim.x;
        uint32_t pos = w - base;
        if (round & 1u) pos = min(gridDim.x, p.n_items - base) - 1u - pos;
        const uint32_t rank = base + pos;
        const uint32_t hb = p.n_items / p.n_qtiles;
        x = p.n_qtiles - 1u - rank / hb;
        yz = rank % hb;
    }
    it.row0 = x * (kRows >> ps);
    const uint32_t hg = p.H >> ps;
    it.head = (yz % hg) << ps;
    const uint32_t z = yz / hg;
    it.batch = z;
    it.split = 0;
    if (kSplit) {
        it.batch = z >> p.split_log2;
        it.split = z & (p.splits - 1u);
    }
    it.kv_head = it.head >> p.gqa_shift;   // crates/amdgpu-stage/src/components.rs:8-17
    const uint32_t ntiles_total = (p.SK + kKeys - 1) / kKeys;
    it.key_lo = 0;
    it.key_hi = p.SK;
    if (kSplit) {   // tiles [split*tps, min(ntiles, (split+1)*tps)) (components.rs:58-74)
        const uint32_t tps = (ntiles_total + p.splits - 1) / p.splits;
        const uint32_t tile_lo = it.split * tps;
        const uint32_t tile_hi = min(ntiles_total, tile_lo + tps);
        it.key_lo = tile_lo * kKeys;
        it.key_hi = min(tile_hi * kKeys, p.SK);
    }
    // causal (crates/amdgpu-stage/src/attention/attn3.rs:298-306): row i sees the keys below min(i + SK - S + 1, SK); the item's last row decides
    if (causal) it.key_hi = min(p.SK, it.row0 + (kRows >> ps) + (p.SK - p.S));
    it.n_tiles = (it.key_hi > it.key_lo) ? static_cast<int>((it.key_hi - it.key_lo + kKeys - 1) / kKeys) : 0;
    if (kCluster == kCutAll) {   // every part has a tile: the launcher's rule
        const uint32_t n = static_cast<uint32_t>(it.n_tiles), lo = (n * part) >> p.cut_log2, hi = (n * (part + 1u)) >> p.cut_log2;
        it.key_hi = min(it.key_hi, it.key_lo + hi * kKeys);
        it.key_lo += lo * kKeys;
        it.n_tiles = static_cast<int>(hi - lo);
    }
    if (it.half != 0u) {   // whole tiles [0, ceil(n / 2)) to the first half, the rest (and a ragged end) to the second
        const int first = (it.n_tiles + 1) / 2;
        if (it.half == 1u) {
            it.key_hi = it.key_lo + static_cast<uint32_t>(first) * kKeys;
            it.n_tiles = first;
        } else {
            it.key_lo += static_cast<uint32_t>(first) * kKeys;
            it.n_tiles -= first;
        }
    }
    return it;
}

}  // namespace

// Persistent: gridDim.x CTAs (one per SM) walk the work items w = blockIdx.x, blockIdx.x + gridDim.x, ... The K / V rings, the score and P
// buffers and every barrier run on one tile counter g that keeps counting across items, so the next item's Q, K and V loads and its first
// two score tiles overlap the current item's last tiles and epilogue; only O is single: P V of an item's first tile waits until the
// epilogue of the item before has read O out (o_free).
// kTrace = false compiles every diagnostic (tile dumps, time stamps) out of the tile loop: the production launches use that variant.
// kLazy: the long-sequence softmax recipe. kCausal: the causal mask (never with kSplit). kCluster: only with kLazy.
// kPack: AttnParams::pack_shift may be set. The row and head arithmetic of it cost 0.5 us an item where items are short, so the other launches have a
// variant without.
// kFused: the split kernel with the merge of the partials built into its epilogue (no pairs, no diagnostics, f16 partials, no peer routing).
template <bool kSplit, bool kTrace, bool kLazy, bool kCausal, Cluster kCluster, bool kVbs, bool kFused = false, bool kPack = kCluster != kNoCluster>
__global__ void __maxnreg__(kMaxRegs)
mxfp8_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const AttnParams p) {
    auto stamp = [](float* trace, int role, int tile, int slot) { stamp_t<kTrace>(trace, role, tile, slot); };
    constexpr bool kPair = kCluster == kPairs, kCut = kCluster == kCutAll;
    const uint32_t pack_shift = kPack ? p.pack_shift : 0u;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    const uint32_t q_smem = smem_base + SmemLayout::q;
    const uint32_t k_smem = smem_base + SmemLayout::k;
    const uint32_t v_smem = smem_base + SmemLayout::v;
    const uint32_t ones_smem = smem_base + SmemLayout::ones;
    const uint32_t sfq_smem = smem_base + SmemLayout::sfq;
    const uint32_t sfk_smem = smem_base + SmemLayout::sfk;
    const uint32_t bar0 = smem_base + SmemLayout::bars;
    auto bar_q_full = [&](int b) { return bar0 + 8u * b; };
    auto bar_q_empty = [&](int b) { return bar0 + 8u * (2 + b); };
    auto bar_k_full = [&](int st) { return bar0 + 8u * (4 + st); };
    auto bar_k_empty = [&](int st) { return bar0 + 8u * (4 + kStages + st); };
    auto bar_v_full = [&](int st) { return bar0 + 8u * (4 + 2 * kStages + st); };
    auto bar_v_empty = [&](int st) { return bar0 + 8u * (4 + 3 * kStages + st); };
    auto bar_s_full = [&](int b) { return bar0 + 8u * (4 + 4 * kStages + b); };
    auto bar_s_free = [&](int b) { return bar0 + 8u * (6 + 4 * kStages + b); };
    auto bar_p_full = [&](int b) { return bar0 + 8u * (8 + 4 * kStages + b); };
    auto bar_o_done = [&](int b) { return bar0 + 8u * (10 + 4 * kStages + b); };
    const uint32_t bar_o_free = bar0 + 8u * (12 + 4 * kStages);
    const uint32_t bar_o_full = bar0 + 8u * (13 + 4 * kStages);
    // pairs: "this CTA's exchange area is free" (one arrival, from the partner with the first half) and "the partner's half item has
    // landed in this CTA's exchange area" (128 arrivals, from the partner with the second half)
    const uint32_t bar_peer_rdy = bar0 + 8u * (18 + 4 * kStages), bar_peer_data = bar0 + 8u * (19 + 4 * kStages);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + SmemLayout::tmem_slot);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + SmemLayout::abort_flag);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n_items = p.n_work, stride = gridDim.x;   // the work units this grid walks (whole items, and halves of the last round's)
    // kLazy: the long-sequence recipe, chosen by the launcher from the whole sequence's tile count, also in a split (block3.rs:180-184)
    constexpr bool lazy = kLazy;
    const bool cta_traced = kTrace && p.trace != nullptr && blockIdx.x == 0;   // diagnostics cover the first item of CTA 0 = logical block (0,0,0)

    // Programmatic dependent launch: the next launch in the stream (if it asks for it, as this library's own launches do) may be
    // scheduled while this grid runs; its CTAs become resident as ours exit and do their set-up, then wait below for this grid's end.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // ---- one-time setup ----
    if (threadIdx.x == 0) stamp(cta_traced ? p.trace : nullptr, 2, 30, 0);   // kernel entry
    // The producers' copies of scale bytes: E8M0 words of 128 rows -> [row % 32][row / 32][4], the layout tcgen05.cp 32x128b.warpx4 spreads over the four lane
    // quadrants. Lane l copies rows l, l + 32, ...; the copies arrive on the tile's barrier when they have landed (32 arrivals).
    auto copy_q_scales = [&](const Item& it, uint32_t qb) {
        const uint32_t dst = sfq_smem + qb * kSfBytes + static_cast<uint32_t>(lane) * 16u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lr = lane + 32 * i;
            const uint32_t r = min(it.row0 + (lr >> pack_shift), p.S - 1u);   // rows past the sequence reuse the last row's scales (block3.rs:110-113)
            const uint32_t head = it.head + (lr & ((1u << pack_shift) - 1u));
            cp_async_4(dst + 4u * i, p.q_descale + static_cast<size_t>(it.batch) * p.qs_batch_stride + (static_cast<size_t>(r) * p.H + head) * 4u, 4u);
        }
        cp_async_arrive(bar_q_full(qb));
    };
    // `src`: the scale word of this lane's first key of the tile; `keys_left`: sequence keys from there on (keys past the sequence: zeros; their data is zero-filled too)
    auto copy_k_scales = [&](const uint8_t* src, int keys_left, int st) {
        const uint32_t dst = sfk_smem + static_cast<uint32_t>(st) * kSfBytes + static_cast<uint32_t>(lane) * 16u;
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async_4(dst + 4u * i, src + static_cast<size_t>(i) * (32u * p.HK * 4u), 32 * i < keys_left ? 4u : 0u);
        cp_async_arrive(bar_k_full(st));
    };
    auto k_scales_of = [&](const Item& it) { return p.k_descale + static_cast<size_t>(it.batch) * p.ks_batch_stride + (static_cast<size_t>(it.key_lo + lane) * p.HK + it.kv_head) * 4u; };
    // Launched as clusters (items are cut between their CTAs): the partner's barriers must exist before anything can arrive on them. Every thread arrives on
    // the cluster's barrier in the set-up, the warp that sets the barriers up behind that, all in front of the wait for the grid before, and waits for it only where it
    // first touches the partner (the epilogue warpgroup, the score MMA warp) or, failing that, at the end; by then the partner has long arrived. Behind
    // that wait the arrivals stand in every launch's way (back to back: B1 H8 HK2 S512 Skv4096 cut in 8 16.4 us, so 15.9; B1 H10 S2048 Skv8192 as pairs 67.5 and 67.2).
    constexpr bool paired = kCluster != kNoCluster;
    auto arrive_cluster = [&]() {
        if (paired) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    };
    if (warp != kKProducerWarp) arrive_cluster();
    if (warp == kKProducerWarp) {
        // This warp sets the barriers up and sends out the CTA's first copies (Q, K and V tile of its first item, their scales) while the others are still at
        // the rest of the set-up: what a launch starts with is the wait for them. From the role's own loop they went out 600 clocks later (launches in a graph:
        // B1 H2 S256 5.83 us, so 5.42; one row block of 16 tiles 13.30 and 12.86; calls of the former one by one wait for the host, 7.0 us either way).
        if (lane < 3) prefetch_tmap(lane == 0 ? &tm_q : lane == 1 ? &tm_k : &tm_v);
        const uint32_t l = static_cast<uint32_t>(lane);
        uint32_t count = 1u;                                   // of barrier l (SmemLayout::bars); lanes 30 and 31: peer_rdy and peer_data
        if (l < 2u || (l >= 4u && l < 8u)) count = 1u + 32u;     // q_full, k_full: the TMA's expect-tx arrive + the producer lanes' scale copies
        if (kVbs && l >= 12u && l < 16u) count = 2u;             // v_full: the same + the arrive that follows V's scale bytes
        if (l >= 22u && l < 26u) count = kRows;                  // s_free, p_full
        if (l == 28u || l == 31u) count = kRows;                 // o_free (the epilogue warpgroup's 128 threads), peer_data
        if (l == 30u) count = kCut ? 1u << p.cut_log2 : 1u;
        static_assert(kStages == 4, "the barriers' order");
        mbar_init(bar0 + 8u * (l < 30u ? l : l + 4u), count);
        if (lane == 0) *abort_flag = 0u;
        fence_mbar_init();
        __syncwarp();
        arrive_cluster();
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (see below)
        if (blockIdx.x < n_items) {
            const Item it = decode_item<kSplit, kCausal, kCluster, kPack>(blockIdx.x, p);
            if (elect_one_sync()) {
                mbar_arrive_expect_tx(bar_q_full(0), kTileBytes);
                tma_load_4d(q_smem, &tm_q, bar_q_full(0), 0, static_cast<int>(it.head), static_cast<int>(it.row0), static_cast<int>(it.batch));
                stamp(cta_traced ? p.trace : nullptr, 2, 0, 6);
                mbar_arrive_expect_tx(bar_k_full(0), kTileBytes);
                tma_load_4d(k_smem, &tm_k, bar_k_full(0), 0, static_cast<int>(it.kv_head), static_cast<int>(it.key_lo), static_cast<int>(it.batch));
                stamp(cta_traced ? p.trace : nullptr, 3, 0, 6);
                mbar_arrive_expect_tx(bar_v_full(0), kTileBytes);
                tma_load_4d(v_smem, &tm_v, bar_v_full(0), 0, static_cast<int>(it.kv_head), static_cast<int>(it.key_lo), static_cast<int>(it.batch));
            }
            __syncwarp();
            copy_q_scales(it, 0u);
            copy_k_scales(k_scales_of(it), static_cast<int>(p.SK - it.key_lo) - lane, 0);
        }
    }
    if ((kLazy || kVbs) && threadIdx.x >= 128 && threadIdx.x < 256) {
        reinterpret_cast<uint32_t*>(smem_gen + SmemLayout::sf_one)[threadIdx.x - 128] = 0x7F7F7F7Fu;
        fence_proxy_async_smem();
    }
    if (threadIdx.x >= 256) {
        const uint32_t t = threadIdx.x - 256u;
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint32_t*>(smem_gen + SmemLayout::ones)[t + 256 * i] = 0x38383838u;
        // the 1024 reference hand-over slots start with a tile counter no tile has
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint2*>(smem_gen + SmemLayout::xref)[t + 256 * i] = make_uint2(0u, 0xFFFFFFFFu);
        reinterpret_cast<uint32_t*>(smem_gen + SmemLayout::sfp)[t] = 0x7F7F7F7Fu;
        fence_proxy_async_smem();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    bool cluster_joined = !paired;
    auto join_cluster = [&]() {
        if (!cluster_joined) {
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            cluster_joined = true;
        }
    };
    // nothing above but the first copies, which wait for themselves, touches global memory; everything below may read what the previous grid in the stream wrote
    // (a quantiser that is still writing the scales as this grid starts, for one): by TMA, cp.async or ld in volatile asm, which stays behind the wait, never through __ldg, which the
    // compiler may move in front of it
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x == 0) stamp(cta_traced ? p.trace : nullptr, 2, 30, 2);   // setup done

    // The four service roles are single chains of dependent instructions that share their scheduler with four arithmetic-dense softmax
    // warps, so every instruction costs them several clocks: each role is its own warp, waits with blocking mbarrier waits (its
    // conditions are conjunctions, never alternatives) and keeps its per-tile instruction count small.
    // The register file is split unevenly: the kernel starts with kMaxRegs registers in every thread; the four service warps (one
    // warpgroup) give most of theirs back and the softmax warpgroups take them, which lets the compiler keep the whole score row plus
    // enough temporaries to interleave the conversion's dependent chains without spilling (4-6 % on the full machine).
    if (warp < kFirstSoftmaxWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kServiceRegs));
    if (warp == kKProducerWarp || warp == kVProducerWarp) {
        // =========================================================== producers: Q, K, V tiles; Q and K scales ===========================================================
        // Warp 1 issues the Q and K tile copies and, with 4-byte asynchronous copies, their scale bytes (4 per row, strided by the head count, which a
        // TMA box cannot express); warp 3 issues the V tile copies. Both run ahead as far as their rings go, and neither's tiles wait for the other's ring: with a K
        // tile's scales behind the V ring on every second tile, as loads into registers four tiles ahead, B2 H16 HK4 S1000 Skv1337 took 21.8 us, so 19.2;
        // B1 H8 S2048 16.5 and 14.9; B4 H8 S2048 50.7 and 49.8 (back to back; the set-up's first copies have their share in it).
        auto producer = [&](auto is_k_c) {
            constexpr bool kIsK = decltype(is_k_c)::value;
            const uint32_t tile_step = 128u * p.HK * 4u;   // of the K scales: bytes between key tiles
            uint32_t g = 0, n = 0, ph = 0, q_issued = 0;   // g: the running tile counter
            int st = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; ok && w < n_items; w += stride, ++n) {
                const Item it = decode_item<kSplit, kCausal, kCluster, kPack>(w, p);
                const uint32_t qb = n & 1u;
                if (kIsK) {
                    // the Q buffer was last used two items ago
                    if (n >= 2) ok = mbar_wait(bar_q_empty(qb), ((n >> 1) - 1u) & 1u, abort_flag);
                    if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
                    if (n > 0 && elect_one_sync()) {
                        mbar_arrive_expect_tx(bar_q_full(qb), kTileBytes);
                        tma_load_4d(q_smem + qb * kTileBytes, &tm_q, bar_q_full(qb), 0, static_cast<int>(it.head), static_cast<int>(it.row0), static_cast<int>(it.batch));
                    }
                    if (n > 0) copy_q_scales(it, qb);
                    ++q_issued;
                }
                const uint8_t* k_scales = k_scales_of(it);
                int keys_left = static_cast<int>(p.SK - it.key_lo) - lane;
                float* k_trace = cta_traced ? p.trace : nullptr;   // stamps are indexed by the running tile counter
                int key = static_cast<int>(it.key_lo);
                for (int j = 0; j < it.n_tiles; ++j, key += kKeys) {
                    uint32_t vsc[4] = {0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu};   // key blocks past the sequence: data is zero-filled, any finite scale does
                    if (kVbs && !kIsK) {   // issued first, used after the waits below
                        const uint32_t nblk = (p.SK + 31u) / 32u, blk0 = static_cast<uint32_t>(key) / 32u;
#pragma unroll
                        for (uint32_t kb = 0; kb < 4u; ++kb) {
                            ld_global_u32_if(vsc[kb], p.v_blockscale + ((static_cast<size_t>(it.batch) * nblk + blk0 + kb) * p.HK + it.kv_head) * 128u + 4u * static_cast<uint32_t>(lane), blk0 + kb < nblk);
                        }
                    }
                    // K: the stage (tile and scale bytes) is free once Q K^T of the tile that held it is done
                    if (kIsK) {
                        if (g >= static_cast<uint32_t>(kStages)) ok = mbar_wait(bar_k_empty(st), ph ^ 1u, abort_flag);
                        if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
                        if (g > 0 && elect_one_sync()) {
                            stamp(k_trace, 2, static_cast<int>(g), 6);
                            mbar_arrive_expect_tx(bar_k_full(st), kTileBytes);
                            tma_load_4d(k_smem + st * kTileBytes, &tm_k, bar_k_full(st), 0, static_cast<int>(it.kv_head), key, static_cast<int>(it.batch));
                        }
                        if (g > 0) copy_k_scales(k_scales, keys_left, st);   // (the CTA's first tile, and the first item's Q, went out in the set-up)
                        k_scales += tile_step;
                        keys_left -= kKeys;
                    }
                    if (!kIsK) {
                        // V: the stage is free once P V of the tile that held it is done
                        if (g >= static_cast<uint32_t>(kStages)) ok = mbar_wait(bar_v_empty(st), ph ^ 1u, abort_flag);
                        if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
                        if (g > 0 && elect_one_sync()) {
                            stamp(k_trace, 3, static_cast<int>(g), 6);
                            mbar_arrive_expect_tx(bar_v_full(st), kTileBytes);
                            tma_load_4d(v_smem + st * kTileBytes, &tm_v, bar_v_full(st), 0, static_cast<int>(it.kv_head), key, static_cast<int>(it.batch));
                        }
                        if (kVbs) {
                            // V block scales (extension): E8M0 [batch][key / 32][kv head][128 columns]. The tile's four key blocks are four rows of
                            // 128 bytes; lane l holds columns 4l .. 4l+3 of each (vsc, loaded at the top of the iteration), transposes them to
                            // one word per column (byte = key block) and writes word n to [n % 32][n / 32], the layout tcgen05.cp spreads
                            // over the lane quadrants.
                            const uint32_t a0 = __byte_perm(vsc[0], vsc[1], 0x5140), a1 = __byte_perm(vsc[0], vsc[1], 0x7362);
                            const uint32_t b0 = __byte_perm(vsc[2], vsc[3], 0x5140), b1 = __byte_perm(vsc[2], vsc[3], 0x7362);
                            const uint32_t t[4] = {__byte_perm(a0, b0, 0x5410), __byte_perm(a0, b0, 0x7632), __byte_perm(a1, b1, 0x5410), __byte_perm(a1, b1, 0x7632)};
                            uint32_t* sfv_dst = reinterpret_cast<uint32_t*>(smem_gen + SmemLayout::sfv + st * kSfBytes);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t n = 4u * static_cast<uint32_t>(lane) + static_cast<uint32_t>(i);
                                sfv_dst[(n & 31u) * 4u + (n >> 5)] = t[i];
                            }
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (elect_one_sync()) mbar_arrive(bar_v_full(st));
                        }
                    }
                    ++g;
                    if (++st == kStages) { st = 0; ph ^= 1u; }
                }
            }
            cp_async_wait_all();
            if (*abort_flag != 0u) {
                // leaving early: let the tile copies already in flight land before the CTA's shared memory is given back
                for (uint32_t t = g > static_cast<uint32_t>(kStages) ? g - kStages : 0u; t < g; ++t) {
                    const long long t0 = clock64();
                    while (!mbar_test_wait(kIsK ? bar_k_full(t % kStages) : bar_v_full(t % kStages), (t / kStages) & 1u) && clock64() - t0 < kWaitBudgetCycles) {}
                }
                for (uint32_t m = q_issued > 2u ? q_issued - 2u : 0u; m < q_issued; ++m) {
                    const long long t0 = clock64();
                    while (!mbar_test_wait(bar_q_full(m & 1u), (m >> 1) & 1u) && clock64() - t0 < kWaitBudgetCycles) {}
                }
            }
        };
        if (warp == kKProducerWarp) producer(std::true_type{});
        else producer(std::false_type{});
    } else if (warp == kMmaWarp) {
        // =========================================================== MMA issuer: score tiles ===========================================================
        // The whole warp runs the role in step on warp-uniform values and an elected lane issues: written as `if (lane == 0) { ... }` the
        // role spent 400 clocks per tile on issuing four MMAs and 200 on the commits, because every operand of a tcgen05 instruction then
        // has to be moved over from vector registers; now 120 and 45. Q K^T and P V are issued by two different threads (this warp's and
        // kPvWarp's elected lanes): their streams share no operand, the pipe interleaves them, and neither holds the other up.
        {
            const uint32_t idesc_qk = idesc_mxf8_block_scaled(128, 128, 0, 0, 0, 0);
            const uint32_t t_sfq = tmem + kColSfQ;
            // K-major 128-byte-swizzled Q / K tiles: 8-row groups 1024 B apart, 32 head-dim bytes (two 16-byte units) per MMA
            const uint64_t dq0 = make_smem_desc(q_smem, 16, 1024, kSwizzle128B);
            const uint64_t dk0 = make_smem_desc(k_smem, 16, 1024, kSwizzle128B);
            const uint64_t dsf0 = make_smem_desc(sfk_smem, 0, 128, kSwizzleNone);
            const uint64_t dsfq0 = make_smem_desc(sfq_smem, 0, 128, kSwizzleNone);
            uint32_t g = 0, n = 0, ph = 0;
            int st = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; ok && w < n_items; w += stride, ++n) {
                const Item qk_it = decode_item<kSplit, kCausal, kCluster, kPack>(w, p);
                const int n_tiles = qk_it.n_tiles;
                const uint32_t qb = n & 1u;
                float* mma_trace = cta_traced ? p.trace : nullptr;
                // first half of a cut item: once its last score tile is done the K ring is idle for good, and the partner may push its
                // half there (the commit below arrives on the partner's barrier)
                if (kCut) join_cluster();   // (the same with the other CTAs of the cluster)
                uint32_t partner_rdy = 0u;
                if (kPair && qk_it.half == 1u) {
                    join_cluster();
                    partner_rdy = map_to_cta(bar_peer_rdy, 1u);
                }
                ok = mbar_wait(bar_q_full(qb), (n >> 1) & 1u, abort_flag);
                if (!ok) break;
                tc_fence_after_sync();
                fence_proxy_async_smem();   // the scale bytes are written by the producer lanes' asynchronous copies (generic writes, acquired by the wait) and read by tcgen05.cp
                // issued behind the previous item's MMAs by the same thread, so it cannot overtake their reads of these columns
                if (elect_one_sync()) tmem_cp_sf(t_sfq, dsfq0 + static_cast<uint64_t>((qb * kSfBytes) >> 4));
                const uint64_t dq = dq0 + static_cast<uint64_t>((qb * kTileBytes) >> 4);
                for (int j = 0; j < n_tiles; ++j) {
                    // S[g&1] = Q K(j)^T: needs the K tile and its scales, and the softmax of tile g-2 to have read S[g&1] out
                    ok = mbar_wait(bar_k_full(st), ph, abort_flag);
                    if (ok && g >= 2) ok = mbar_wait(bar_s_free(g & 1u), ((g >> 1) - 1u) & 1u, abort_flag);
                    if (!ok) break;
                    fence_proxy_async_smem();   // (the K scales' copies are generic writes too)
                    tc_fence_after_sync();
                    if (lane == 0) stamp(mma_trace, 2, static_cast<int>(g), 2);
                    const uint32_t t_sfk = tmem + ((g & 1u) ? kColSfK1 : kColSfK0);
                    const uint32_t t_s = tmem + ((g & 1u) ? kColS1 : kColS0);
                    const uint64_t dk = dk0 + static_cast<uint64_t>((st * kTileBytes) >> 4);
                    if (elect_one_sync()) {
                        tmem_cp_sf(t_sfk, dsf0 + static_cast<uint64_t>((st * kSfBytes) >> 4));
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb) {
                            const uint32_t id = idesc_qk | (static_cast<uint32_t>(kb) << 29) | (static_cast<uint32_t>(kb) << 4);
                            mma_mxf8_ss(t_s, dq + 2u * kb, dk + 2u * kb, id, t_sfq + (static_cast<uint32_t>(kb) << 30),
                                        t_sfk + (static_cast<uint32_t>(kb) << 30), kb > 0 ? 1u : 0u);
                        }
                        stamp(mma_trace, 2, static_cast<int>(g), 4);
                        tc_commit(bar_s_full(g & 1u));
                        tc_commit(bar_k_empty(st));
                        if (j == n_tiles - 1) tc_commit(bar_q_empty(qb));   // the Q buffer can take the item after next
                        if (kPair && partner_rdy != 0u && j == n_tiles - 1) tc_commit(partner_rdy);
                        if (kCut && j == n_tiles - 1) {
                            for (uint32_t c = 0; c < (1u << p.cut_log2); ++c) tc_commit(map_to_cta(bar_peer_rdy, c));
                        }
                        stamp(mma_trace, 2, static_cast<int>(g), 5);
                    }
                    ++g;
                    if (++st == kStages) { st = 0; ph ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == kPvWarp) {
        // =========================================================== MMA issuer: P V ===========================================================
        {
            // P V with N = 144: head dims 0..127 from the V tile, 16 more columns from the tile of ones (O | L are adjacent in TMEM)
            const uint32_t idesc_pv = idesc_f8_dense(128, 144, 0, 1);
            // V block scales (extension): the same MMA as kind::mxf8f6f4.block_scale, P's factors a constant 1.0, V's one E8M0 per 32 keys and column
            const uint32_t idesc_pv_bs = idesc_mxf8_block_scaled(128, 144, 0, 1, 0, 0);
            const uint32_t t_sfp = tmem + kColSfP, t_sfv = tmem + kColSfV;
            constexpr bool kScaled = kLazy || kVbs;   // P V as the block-scaled kind
            if (kScaled && elect_one_sync()) {   // the constant factors, once: the ones columns' (rows 128..143 of the B factors), V's without block scales, P's in the short recipe
                const uint64_t d1 = make_smem_desc(smem_base + SmemLayout::sf_one, 0, 128, kSwizzleNone);
                if (!kLazy) tmem_cp_sf(t_sfp, d1);
                if (!kVbs) tmem_cp_sf(t_sfv, d1);
                tmem_cp_sf(t_sfv + 4, d1);
            }
            const uint64_t dsfp0 = make_smem_desc(smem_base + SmemLayout::sfp, 0, 128, kSwizzleNone);
            // MN-major B: 8-key groups 1024 B apart; the second 128-byte-wide atom (columns 128..) is the tile of ones. Moving the start address on moves the
            // distance to the ones back
            const uint64_t dv0 = make_smem_desc(v_smem, ones_smem - v_smem, 1024, kSwizzle128B);
            constexpr uint64_t kDvKeys = (4096u >> 4) - (static_cast<uint64_t>(4096u >> 4) << 16), kDvStage = (kTileBytes >> 4) - (static_cast<uint64_t>(kTileBytes >> 4) << 16);
            uint64_t dv_st = dv0;
            uint32_t g = 0, n = 0, ph = 0;
            int st = 0;
            bool ok = true;
            for (uint32_t w = blockIdx.x; ok && w < n_items; w += stride, ++n) {
                const int n_tiles = decode_item<kSplit, kCausal, kCluster, kPack>(w, p).n_tiles;
                float* mma_trace = cta_traced ? p.trace : nullptr;
                // an item's first tile overwrites O and L, which the epilogue of the item before must have read out
                if (n > 0) ok = mbar_wait(bar_o_free, (n - 1u) & 1u, abort_flag);
                for (int i = 0; ok && i < n_tiles; ++i) {
                    // O (+)= P(i) V(i) with the row sums riding along: P from TMEM (32 columns, 8 per 32 keys), V tile = 128 keys x 128 B, MN-major
                    ok = mbar_wait(bar_v_full(st), ph, abort_flag);
                    if (ok) ok = mbar_wait(bar_p_full(g & 1u), (g >> 1) & 1u, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    if (lane == 0) stamp(mma_trace, 3, static_cast<int>(g), 2);
                    const uint32_t t_p = tmem + ((g & 1u) ? kColP1 : kColP0);
                    if (elect_one_sync()) {
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb) {
                            const uint64_t dv = dv_st + static_cast<uint64_t>(kb) * kDvKeys;
                            if (kScaled) {
                                if (kLazy && kb == 0) tmem_cp_sf(t_sfp, dsfp0 + static_cast<uint64_t>(((g & 1u) * kSfBytes) >> 4));
                                if (kVbs && kb == 0) tmem_cp_sf(t_sfv, make_smem_desc(smem_base + SmemLayout::sfv + st * kSfBytes, 0, 128, kSwizzleNone));
                                const uint32_t id = idesc_pv_bs | (static_cast<uint32_t>(kb) << 29) | (static_cast<uint32_t>(kb) << 4);
                                mma_mxf8_ts(tmem + kColO, t_p + 8 * kb, dv, id, t_sfp + (static_cast<uint32_t>(kb) << 30), t_sfv + (static_cast<uint32_t>(kb) << 30),
                                            (i > 0 || kb > 0) ? 1u : 0u);
                            } else {
                                mma_f8_ts(tmem + kColO, t_p + 8 * kb, dv, idesc_pv, (i > 0 || kb > 0) ? 1u : 0u);
                            }
                        }
                        stamp(mma_trace, 3, static_cast<int>(g), 3);
                        tc_commit(bar_v_empty(st));
                        tc_commit(bar_o_done(g & 1u));
                        if (i == n_tiles - 1) tc_commit(bar_o_full);   // the item's O and L are complete: over to the epilogue warpgroup
                        stamp(mma_trace, 3, static_cast<int>(g), 4);
                    }
                    ++g;
                    dv_st += kDvStage;
                    if (++st == kStages) { st = 0; ph ^= 1u; dv_st = dv0; }
                }
            }
        }
        __syncwarp();
    }
    } else if (warp < kFirstEpilogueWarp) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        // =========================================================== softmax ===========================================================
        // Two warpgroups: wg = parity = which tiles (counter g = parity mod 2) and which S / P buffer. Thread r of a group owns query row r.
        const uint32_t st_id = threadIdx.x - 32u * kFirstSoftmaxWarp;
        const uint32_t wg = st_id >> 7;
        const uint32_t par = wg;
        const uint32_t r = 32u * (static_cast<uint32_t>(warp) & 3u) + static_cast<uint32_t>(lane);   // TMEM lane = 32 * (warp % 4) + lane
        const uint32_t lane_base = (static_cast<uint32_t>(warp & 3) * 32u) << 16;
        const uint32_t xref = smem_base + SmemLayout::xref;   // 8-byte slots, accessed with single 64-bit shared loads / stores
        const uint32_t t_s = tmem + (par ? kColS1 : kColS0) + lane_base;
        const uint32_t t_p = tmem + (par ? kColP1 : kColP0) + lane_base;
        const uint32_t t_o_part = tmem + kColO + lane_base;
        const uint32_t t_l = tmem + kColL + lane_base;
        bool ok = true;

        // bounded poll of an 8-byte {value, tile counter} slot
        auto wait_slot = [&](uint32_t slot, uint32_t g, float& out) -> bool {
            uint2 o = ld_shared_v2(slot);
            if (o.y != g) {
                const long long t0 = clock64();
                for (uint32_t spins = 1;; ++spins) {
                    o = ld_shared_v2(slot);
                    if (o.y == g) break;
                    if ((spins & 15u) == 0u && (*abort_flag != 0u || clock64() - t0 > kWaitBudgetCycles)) { *abort_flag = 1u; return false; }
                }
            }
            out = __uint_as_float(o.x);
            return true;
        };
        // what tile g did to the row's reference, published by the thread that handled it
        auto ref_slot = [&](uint32_t g) { return xref + 8u * ((g & 7u) * 128u + r); };

        // Long-sequence recipe: P of a tile is handed over under the next tile's tensor-memory round trip (or when the role ends): the wait for its stores is then
        // free
        bool p_ready = false;
        auto hand_over_p = [&]() {
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive_if(bar_p_full(par), p_ready);
            p_ready = false;
        };
        const bool want_fin = kSplit || p.lse_nat != nullptr || cta_traced || kCluster != kNoCluster;   // does anything read the final reference?
        float sf_held = 0.0f;   // log2 of the four block scales this group's buffer holds for the row, if they are equal
        auto scale_o = [&](float f) {
#pragma unroll 1
            for (int c = 0; c < 2; ++c) scale_tmem64(t_o_part + 64 * c, f);
            uint32_t lv;   // the row sum lives in column 0 of L
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(lv) : "r"(t_l) : "memory");
            tmem_wait_ld();
            lv = __float_as_uint(__uint_as_float(lv) * f);
            asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(t_l), "r"(lv) : "memory");
        };
        uint32_t g0 = 0, n = 0;   // tile counter at the item's first tile; ordinal of the item
        for (uint32_t w = blockIdx.x; ok && w < n_items; w += stride, ++n) {
            // the tile count, the number of tiles every row sees in full and the row's own key limit stay live through the tile loop
            int n_tiles, j_full, row_lim;   // row_lim: this row's visible keys, counted from the item's first key
            {
                const Item it = decode_item<kSplit, kCausal, kCluster, kPack>(w, p);
                n_tiles = it.n_tiles;
                row_lim = static_cast<int>(it.key_hi - it.key_lo);
                int first_lim = row_lim;   // the limit of the item's first row: the tiles below it need no mask
                if (kCausal && !kSplit) {
                    const int visible = static_cast<int>(it.row0 + 1u + (p.SK - p.S)) - static_cast<int>(it.key_lo);   // to the item's first row; none (<= 0) in a part behind its diagonal
                    first_lim = max(min(row_lim, visible), 0);
                    row_lim = min(row_lim, visible + static_cast<int>(r >> pack_shift));
                }
                j_full = first_lim / kKeys;
            }
            const bool tracing = cta_traced && n == 0;
            const bool dumping = tracing && !(p.flags & 0x4u);   // flag 0x4: time stamps only, no tile dumps
            float ref = lazy ? kNoRef : -INFINITY;   // the row's reference (log2 units) after the last tile this thread has seen
            float base = -INFINITY;  // long-sequence recipe: what the row's O and L are in units of

            uint32_t v[128];         // the row's scores of a tile, converted in place
            uint32_t pw[kCols / 4];  // the row's P words
            auto chunk = [&](int ch) -> uint32_t(&)[32] { return *reinterpret_cast<uint32_t(*)[32]>(&v[32 * ch]); };
            auto mask_scores = [&](int j) {   // keys past the range: -inf for the maximum, 0 for P (crates/amdgpu-tile/src/reduce.rs:35-49)
                const int valid = row_lim - j * kKeys;   // may be <= 0 on the causal diagonal: the row then has no key in this tile
#pragma unroll
                for (int c = 0; c < 128; ++c) {
                    if (c >= valid) v[c] = 0xFF800000u;
                }
            };

            // ---- the long-sequence recipe
            // Every block of 32 keys has a reference of its own: P = 2^(s - ref + offset) in e4m3, and its P V goes into O with the block scale
            // 2^(ref - base) on P (one E8M0 per row and 32 keys of the A operand); base is the row's reference after its first tile. So O is not rescaled
            // when a row's maximum grows, and no group waits for the other one's reference. O and the row sums are in units of
            // 2^(base - offset), in f32; only a row that grows by more than kRebase binades past its base (f32 has room for twice that) gets a
            // new base, and O and L are then rescaled in tensor memory.
            // A block's reference is the one before it (of this group's last tile, or of the other group's tile before that if that is higher), or
            // ceil(block maximum) if the maximum passes that by more than the threshold: an integer that only grows, within an item or (ref_mask) a run of
            // its tiles.
            // The maximum of block b + 1 is taken while block b is converted. The conversion is a software pipeline over the 32 words: word c's
            // exp2 (two values) and bit-built values (two) are started kConvDepth words before they are packed.
            auto tile_lazy = [&](int j, auto masked_c) {
                constexpr bool kMasked = decltype(masked_c)::value;
                const uint32_t g = g0 + static_cast<uint32_t>(j);
                const uint32_t k = g >> 1;   // this parity's tile counter
                float* st_trace = (cta_traced && r == 0) ? p.trace : nullptr;
                const uint32_t j_seg = static_cast<uint32_t>(j) & p.ref_mask;   // tile within its run of tiles that share a reference
                if (j_seg < 2u) ref = kNoRef;                                   // this group's first tile of the run
                stamp(st_trace, par, static_cast<int>(g), 0);
                if (!mbar_wait(bar_s_full(par), k & 1u, abort_flag)) ok = false;   // no divergent exit: a failed wait only clears `ok`, the vote after the tile loop ends the role
                tc_fence_after_sync();
                stamp(st_trace, par, static_cast<int>(g), 1);
                tmem_ld32(t_s, chunk(0));
                hand_over_p();
                tmem_wait_ld();
                reg_fence32(chunk(0));
#pragma unroll
                for (int ch = 1; ch < 4; ++ch) tmem_ld32(t_s + 32 * ch, chunk(ch));
                if (kMasked) {
                    tmem_wait_ld();
#pragma unroll
                    for (int ch = 1; ch < 4; ++ch) reg_fence32(chunk(ch));
                    mask_scores(j);
                }
                float m[4] = {}, refs[4], sh = 0.0f, cf = 0.0f;
                auto max_words = [&](int c) {   // two words, four independent chains
                    m[0] = max3(m[0], __uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1]));
                    m[1] = max3(m[1], __uint_as_float(v[4 * c + 2]), __uint_as_float(v[4 * c + 3]));
                    m[2] = max3(m[2], __uint_as_float(v[4 * c + 4]), __uint_as_float(v[4 * c + 5]));
                    m[3] = max3(m[3], __uint_as_float(v[4 * c + 6]), __uint_as_float(v[4 * c + 7]));
                };
                auto max_reset = [&]() { m[0] = m[1] = m[2] = m[3] = -INFINITY; };
                auto next_reference = [&](int b) {
                    const float mt = fmaxf(max3(m[0], m[1], m[2]), m[3]);
                    if (mt - kLazyThreshold > ref) ref = ceilf(mt);
                    refs[b] = ref;
                };
                auto use_reference = [&](int b) {
                    sh = kPOffset - refs[b];
                    cf = (kPOffset + 7.0f - kFastBias - refs[b]) * 0x1p-21f;
                };
                constexpr int kConvDepth = 8;
                auto conv_start = [&](int c) {
                    add2(v[4 * c], v[4 * c + 1], sh);
                    v[4 * c] = __float_as_uint(ex2_approx(__uint_as_float(v[4 * c])));
                    v[4 * c + 1] = __float_as_uint(ex2_approx(__uint_as_float(v[4 * c + 1])));
                    fma2(v[4 * c + 2], v[4 * c + 3], 0x1p-21f, cf);
                };
                auto conv_finish = [&](int d) {
                    const uint32_t lo = cvt_e4m3x2(__uint_as_float(v[4 * d]), __uint_as_float(v[4 * d + 1]));
                    pw[d] = __byte_perm(lo, cvt_relu_f16x2(__uint_as_float(v[4 * d + 2]), __uint_as_float(v[4 * d + 3])), 0x6410);
                };
                if (dumping && j == 0) {
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 128; ++c) p.trace[r * 128 + c] = __uint_as_float(v[c]);
                }
                max_reset();
#pragma unroll
                for (int c = 0; c < 8; c += 2) max_words(c);
                next_reference(0);
                use_reference(0);
                if (!kMasked) {
                    tmem_wait_ld();
#pragma unroll
                    for (int ch = 1; ch < 4; ++ch) reg_fence32(chunk(ch));
                }
                // the scores are in registers: Q K^T of tile g + 2 may overwrite them
                tc_fence_before_sync();
                mbar_arrive(bar_s_free(par));
                stamp(st_trace, par, static_cast<int>(g), 2);
                bool pv_seen = false;
                uint2 prev = make_uint2(0u, g);   // (tag g: not the one looked for)
#pragma unroll
                for (int c = 0; c < 32 + kConvDepth; ++c) {
                    if (c % 8 == 0 && c > 0 && c < 32) use_reference(c / 8);
                    if (c < 32) conv_start(c);
                    if (c < 24) {
                        if (c % 8 == 0) max_reset();
                        if (c % 2 == 0) max_words(c + 8);
                        if (c % 8 == 7) next_reference(c / 8 + 1);
                    }
                    if (c == 24) {
                        st_shared_v2(ref_slot(g), __float_as_uint(ref), g);
                        pv_seen = mbar_test_wait(bar_o_done(par), (k - 1u) & 1u);   // probed ahead: P V of this parity's previous tile (true for the first: the phase before a new barrier's)
                    }
                    if (c == 32 && j > 0) prev = ld_shared_v2(ref_slot(g - 1u));
                    if (c >= kConvDepth) conv_finish(c - kConvDepth);
                }
                if (dumping && j == 0) {
#pragma unroll
                    for (int c = 0; c < kCols / 4; ++c) reinterpret_cast<uint32_t*>(p.trace)[32768 + 256 + r * 32 + c] = pw[c];
                }
                stamp(st_trace, par, static_cast<int>(g), 5);
                // The row's base after the previous tile and after this one. Both groups follow the published references with the same rule, so
                // they agree on it; the reference of the previous tile was published a tile's time ago
                float ref_prev = __uint_as_float(prev.x), base_prev = base;
                if (j > 0) {
                    if (prev.y != g - 1u && ok && !wait_slot(ref_slot(g - 1u), g - 1u, ref_prev)) ok = false;
                    if (ref_prev - base > kRebase<kVbs>) base_prev = ref_prev;
                } else {
                    base_prev = ref;
                }
                base = ref - base_prev > kRebase<kVbs> ? ref : base_prev;
                const bool rebase = base != base_prev;
                // P V of this parity's previous tile must be done before its P columns and scales are overwritten (and, observed in order,
                // this keeps the phase parity of the other parity's barrier below unambiguous)
                if (!pv_seen && !mbar_wait(bar_o_done(par), (k - 1u) & 1u, abort_flag)) ok = false;
                // The item's last tile leaves the row's base for the epilogue warpgroup's log-sum-exp: before this thread's arrive
                // on p_full (which the last P V, and through it the epilogue's o_full, come after), and behind the wait above: P V of tile
                // g - 2 is done, so P V of g - 3 is, so the epilogue has taken the item four back out (o_free) and read its slot
                if (want_fin && j == n_tiles - 1) *reinterpret_cast<volatile float*>(smem_gen + SmemLayout::xfin + 4u * ((n & 3u) * 128u + r)) = base;
                stamp(st_trace, par, static_cast<int>(g), 6);
                tmem_st32(t_p, pw);
                // the row's four scale bytes (one per 32 keys), in the pattern that tcgen05.cp spreads over the lane quadrants; they rarely change
                const float above = refs[0] - base;
                if (__builtin_expect(__any_sync(0xFFFFFFFFu, above != sf_held || ref != refs[0] || rebase), 0)) {
                    uint32_t sf[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) sf[b] = __float_as_uint(fmaxf(refs[b] - base, -127.0f) + 8388735.0f);   // E8M0 in the low byte: exponent + 127
                    reinterpret_cast<volatile uint32_t*>(smem_gen + SmemLayout::sfp + par * kSfBytes)[(r & 31u) * 4u + (r >> 5)] =
                        __byte_perm(__byte_perm(sf[0], sf[1], 0x0040), __byte_perm(sf[2], sf[3], 0x0040), 0x5410);
                    sf_held = ref == refs[0] ? above : INFINITY;   // four equal scales, or to be written again
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (j > 0 && __any_sync(0xFFFFFFFFu, rebase)) {
                        if (!mbar_wait(bar_o_done(par ^ 1u), ((g - 1u) >> 1) & 1u, abort_flag)) ok = false;
                        __syncwarp();
                        tc_fence_after_sync();
                        scale_o(rebase ? ex2_approx(base_prev - base) : 1.0f);
                    }
                }
                if (j_seg != 0u) ref = fmaxf(ref, ref_prev);
                p_ready = true;
                stamp(st_trace, par, static_cast<int>(g), 7);
            };

            // ---- the short-sequence recipe: the reference follows every tile's maximum (within a window), O and L are rescaled when it moves
            auto tile_short = [&](int j, bool masked) {
                const uint32_t g = g0 + static_cast<uint32_t>(j);
                const uint32_t k = g >> 1;
                if (!mbar_wait(bar_s_full(par), k & 1u, abort_flag)) ok = false;
                tc_fence_after_sync();
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) tmem_ld32(t_s + 32 * ch, chunk(ch));
                tmem_wait_ld();
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) reg_fence32(chunk(ch));
                if (masked) mask_scores(j);
                tc_fence_before_sync();
                mbar_arrive(bar_s_free(par));
                if (dumping && j == 0) {
#pragma unroll
                    for (int c = 0; c < 128; ++c) p.trace[r * 128 + c] = __uint_as_float(v[c]);
                }
                float m[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) m[i] = -INFINITY;
#pragma unroll
                for (int c = 0; c < 128; c += 2) m[(c / 2) & 7] = max3(m[(c / 2) & 7], __uint_as_float(v[c]), __uint_as_float(v[c + 1]));
                const float mt = fmaxf(fmaxf(max3(m[0], m[1], m[2]), max3(m[3], m[4], m[5])), fmaxf(m[6], m[7]));
                if (ok && j > 0 && !wait_slot(ref_slot(g - 1u), g - 1u, ref)) ok = false;
                // moves when the tile maximum lies above the reference or less than the window below it: f > 1 scales O and L up
                const bool move = mt + kFollowWindow > ref;
                const float f = move ? ex2_approx(ref - mt) : 1.0f;   // 0 on the first tile (old reference -inf)
                ref = move ? mt : ref;
                st_shared_v2(ref_slot(g), __float_as_uint(ref), g);
                const float s0 = kPOffset - ref;
#pragma unroll
                for (int c = 0; c < 32; ++c) pw[c] = p_word(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3], s0);
                if (dumping && j == 0) {
#pragma unroll
                    for (int c = 0; c < kCols / 4; ++c) reinterpret_cast<uint32_t*>(p.trace)[32768 + 256 + r * 32 + c] = pw[c];
                }
                // P V of this parity's previous tile must be done before its P columns are overwritten and before the item's last tile leaves its reference
                if (k > 0 && !mbar_wait(bar_o_done(par), (k - 1u) & 1u, abort_flag)) ok = false;
                if (want_fin && j == n_tiles - 1) *reinterpret_cast<volatile float*>(smem_gen + SmemLayout::xfin + 4u * ((n & 3u) * 128u + r)) = ref;
                tmem_st32(t_p, pw);
                if (j > 0 && __any_sync(0xFFFFFFFFu, move)) {
                    // O holds P V of all the item's tiles before j once the other parity's last P V is done; P V of tile j cannot start before P is handed over
                    if (!mbar_wait(bar_o_done(par ^ 1u), ((g - 1u) >> 1) & 1u, abort_flag)) ok = false;
                    __syncwarp();
                    tc_fence_after_sync();
                    scale_o(f);
                }
                p_ready = true;
                hand_over_p();   // at once: a few tiles are the whole item, and under the next tile's round trip 2 of them (B16 H32 S256) took 25.6 us, so 24.6
            };
            // tiles [0, j_full) have all their keys for every row; behind them come at most two tiles (a ragged end: one; the causal
            // diagonal: up to two), of which this parity owns at most one
            int j = static_cast<int>((g0 ^ par) & 1u);
            if constexpr (lazy) {
                // the loop has no code for keys past the range: with all SMs busy instruction fetch is scarce enough that it would cost 3 %
                for (; j < j_full; j += 2) tile_lazy(j, std::false_type{});
                if (j < n_tiles) tile_lazy(j, std::true_type{});
            } else {
                for (; j < n_tiles; j += 2) tile_short(j, j >= j_full);
            }
            // an item of one tile has no next tile of its own to hide the hand-over under (2 x 8 heads of 1024 rows in eight splits of one tile: 27.0 us without, 26.0 so)
            if (kSplit && lazy && n_tiles == 1) hand_over_p();
            // a failed wait above only clears `ok`; the warp leaves as one
            if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
            g0 += static_cast<uint32_t>(n_tiles);
        }
        hand_over_p();
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
        // =========================================================== epilogue ===========================================================
        // One warpgroup, thread r = TMEM lane r = query row r of the item. It takes an item's O and L out of tensor memory as soon as the
        // item's last P V is done (o_full) and hands the columns back (o_free) before it normalises and stores, so that the softmax
        // warpgroups go straight on with the next item's tiles and the next item's first P V only waits for the read-out.
        // O * v_descale / l (crates/amdgpu-stage/src/attention/state.rs:79-82) leaves through the two 16 KB staging tiles (128-byte
        // swizzle: 16-byte chunk c of row r sits at chunk c ^ (r % 8)) and TMA stores, which also drop the rows past the sequence
        // (block3.rs:194); a thread owns a row, so direct stores would touch 32 different lines per instruction.
        const uint32_t r = 32u * (static_cast<uint32_t>(warp) & 3u) + static_cast<uint32_t>(lane);
        const uint32_t lane_base = (static_cast<uint32_t>(warp & 3) * 32u) << 16;
        const uint32_t t_o = tmem + kColO + lane_base, t_l = tmem + kColL + lane_base;
        const uint32_t stg = smem_base + SmemLayout::ostage;
        const bool issuer = threadIdx.x == 32u * kFirstEpilogueWarp;
        const bool want_fin = kSplit || p.lse_nat != nullptr || cta_traced || kCluster != kNoCluster;
        // Half items (the cut last round; a half item is a CTA's last unit, so its K / V rings are idle once its last P V is done): the CTA
        // with the first half tells its partner when its K ring is free (the commit of its last score tile arrives on the partner's
        // barrier); the partner pushes its unnormalised O (f32), row sums and references there with distributed-shared-memory stores and
        // arrives on the first half's barrier; the first half merges and stores. Both references are integers (long-sequence recipe), so the rescale factors
        // are exact powers of two.
        // exchange area = the K ring (64 KB): row r at r * 512 bytes, its 16-byte chunk c at position c ^ (r % 8) within each group of 8
        const uint32_t xch_row = smem_base + SmemLayout::k + r * 512u;
        const uint32_t xch_stat = smem_base + SmemLayout::xstat + r * 8u;
        static_assert(128u * 512u <= kStages * kTileBytes, "the exchange area is the K ring");
        auto xch_off = [&](int c, int q4) { return static_cast<uint32_t>(c) * 128u + ((static_cast<uint32_t>(q4) ^ (r & 7u)) << 4); };
        constexpr uint32_t kEpiBar = 1u;   // named barrier of the 128 epilogue threads
        const float vd = kVbs ? 1.0f : __uint_as_float(ld_global_u32(p.v_descale));   // with V block scales the factors are in the MMA and there is no scalar descale
        uint32_t n = 0;
        bool ok = true;
        for (uint32_t w = blockIdx.x; w < n_items; w += stride, ++n) {
            const Item it = decode_item<kSplit, kCausal, kCluster, kPack>(w, p);
            const bool tracing = cta_traced && n == 0;
            const bool dumping = tracing && !(p.flags & 0x4u);
            float* ep_trace = (cta_traced && r == 0 && n < 6) ? p.trace : nullptr;   // epilogue stamps: P V role's row, tile index 24 + item ordinal, slots 0, 1, 5, 7
            stamp(ep_trace, 3, 24 + static_cast<int>(n), 0);
            ok = mbar_wait(bar_o_full, n & 1u, abort_flag);
            if (issuer && n > 0) bulk_wait_group_read0();   // the previous item's stores have read the staging tiles out
            // one barrier: the staging tiles are free, and the decision to go on is the whole warpgroup's (the named barriers below count
            // all 128 threads, so no warp may leave while a sibling goes on)
            if (!named_bar_all(kEpiBar, 128u, ok)) break;
            tc_fence_after_sync();
            stamp(ep_trace, 3, 24 + static_cast<int>(n), 1);
            uint32_t lv;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(lv) : "r"(t_l) : "memory");
            const float ref_fin = want_fin ? *reinterpret_cast<volatile float*>(smem_gen + SmemLayout::xfin + 4u * ((n & 3u) * 128u + r)) : 0.0f;
            tmem_wait_ld();
            float l = __uint_as_float(lv);
            float ref_out = ref_fin;
            if (kPair && it.half == 2u) {
                // second half: wait for the partner's exchange area, push O, l and the reference, one arrive per thread on its barrier
                join_cluster();
                ok = mbar_wait_cluster(bar_peer_rdy, 0u, abort_flag);
                if (!named_bar_all(kEpiBar, 128u, ok)) break;
                const uint32_t dst_row = map_to_cta(xch_row, 0u);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t o[32];
                    tmem_ld32(t_o + 32 * c, o);
                    tmem_wait_ld();
                    if (c == 3) {
                        tc_fence_before_sync();
                        mbar_arrive(bar_o_free);
                    }
#pragma unroll
                    for (int q4 = 0; q4 < 8; ++q4) {
                        asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst_row + xch_off(c, q4)),
                                     "r"(o[4 * q4]), "r"(o[4 * q4 + 1]), "r"(o[4 * q4 + 2]), "r"(o[4 * q4 + 3]) : "memory");
                    }
                }
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(map_to_cta(xch_stat, 0u)), "f"(l), "f"(ref_fin) : "memory");
                mbar_arrive_remote(map_to_cta(bar_peer_data, 0u));
                continue;
            }
            if (kCut) {
                // Every CTA of the cluster has a part of the item's keys. Row r is finished by CTA r % parts: all parts push the row's O (f32, not
                // normalised), row sum and base there, into the K ring, which is idle in all of them once bar_peer_rdy has completed (the
                // commits behind their last score tiles). A row goes out by its own thread, so its one arrival on the owner's barrier covers it;
                // 128 rows' worth of arrivals is what every owner gets (128 / parts rows from each of the parts).
                // Spreading the rows keeps the exchange at 64 KB in and out of every CTA whatever the number of parts, and rows past the
                // sequence are not sent: a decode step exchanges a few rows.
                const uint32_t lg = p.cut_log2, parts = 1u << lg, me = blockIdx.x & (parts - 1u);
                join_cluster();
                ok = mbar_wait_cluster(bar_peer_rdy, 0u, abort_flag);
                if (!named_bar_all(kEpiBar, 128u, ok)) break;
                auto cut_slot = [&](uint32_t source, uint32_t ro) { return (source << (7u - lg)) + ro; };   // row ro of the owner's, from part `source`
                auto cut_off = [&](uint32_t quad, uint32_t ro) { return (quad >> 3) * 128u + (((quad & 7u) ^ (ro & 7u)) << 4); };   // 4 columns
                {
                    const uint32_t owner = r & (parts - 1u), ro = r >> lg, slot = cut_slot(me, ro);
                    const uint32_t dst = map_to_cta(smem_base + SmemLayout::k + slot * 512u, owner);
                    const bool live = it.row0 + (r >> pack_shift) < p.S;
#pragma unroll
                    for (uint32_t c = 0; c < 4; ++c) {
                        uint32_t o[32];
                        tmem_ld32(t_o + 32 * c, o);
                        tmem_wait_ld();
                        if (live) {
#pragma unroll
                            for (uint32_t q4 = 0; q4 < 8; ++q4) {
                                asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + cut_off(8u * c + q4, ro)),
                                             "r"(o[4 * q4]), "r"(o[4 * q4 + 1]), "r"(o[4 * q4 + 2]), "r"(o[4 * q4 + 3]) : "memory");
                            }
                        }
                    }
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(map_to_cta(smem_base + SmemLayout::xstat + slot * 8u, owner)), "f"(l), "f"(ref_fin) : "memory");
                    mbar_arrive_remote(map_to_cta(bar_peer_data, owner));
                }
                ok = mbar_wait_cluster(bar_peer_data, 0u, abort_flag);
                if (!named_bar_all(kEpiBar, 128u, ok)) break;
                // `parts` threads share an owned row, a thread takes every parts-th group of 4 columns
                const uint32_t et = threadIdx.x - 32u * kFirstEpilogueWarp, ro = et >> lg, c0 = et & (parts - 1u);
                const uint32_t mr = (ro << lg) + me, row = it.row0 + (mr >> pack_shift), head = it.head + (mr & ((1u << pack_shift) - 1u));
                if (row < p.S) {
                    auto stat = [&](uint32_t source) {
                        float2 ps;   // {row sum, base}
                        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(ps.x), "=f"(ps.y) : "r"(smem_base + SmemLayout::xstat + cut_slot(source, ro) * 8u) : "memory");
                        return ps;
                    };
                    // the bases are integers: the weights are exact powers of two (0 for a part without a visible key, whose base is kNoRef)
                    float base = -INFINITY, sum = 0.0f;
                    for (uint32_t c = 0; c < parts; ++c) base = fmaxf(base, stat(c).y);
                    for (uint32_t c = 0; c < parts; ++c) {
                        const float2 ps = stat(c);
                        sum += ps.x * ex2_approx(ps.y - base);
                    }
                    const float fin = vd / sum;
                    const size_t prow = (static_cast<size_t>(it.batch) * p.S + row) * p.H + head + (kSplit ? static_cast<size_t>(it.split) * p.rows_total : 0u);
                    uint8_t* dst = kSplit ? static_cast<uint8_t*>(p.ohat) + prow * 256u
                                          : p.o + static_cast<size_t>(it.batch) * p.o_batch_stride + static_cast<size_t>(row) * p.o_row_stride + static_cast<size_t>(head) * p.o_head_stride;
                    for (uint32_t quad = c0; quad < 32u; quad += parts) {
                        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        for (uint32_t c = 0; c < parts; ++c) {
                            const float f = ex2_approx(stat(c).y - base);
                            float4 pb;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(pb.x), "=f"(pb.y), "=f"(pb.z), "=f"(pb.w)
                                         : "r"(smem_base + SmemLayout::k + cut_slot(c, ro) * 512u + cut_off(quad, ro)) : "memory");
                            acc.x = fmaf(pb.x, f, acc.x);
                            acc.y = fmaf(pb.y, f, acc.y);
                            acc.z = fmaf(pb.z, f, acc.z);
                            acc.w = fmaf(pb.w, f, acc.w);
                        }
                        uint2 wv;
                        if (kSplit) {
                            asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(wv.x) : "f"(acc.y * fin), "f"(acc.x * fin));
                            asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(wv.y) : "f"(acc.w * fin), "f"(acc.z * fin));
                        } else {
                            const __nv_bfloat162 b01 = __floats2bfloat162_rn(acc.x * fin, acc.y * fin), b23 = __floats2bfloat162_rn(acc.z * fin, acc.w * fin);
                            wv = make_uint2(*reinterpret_cast<const uint32_t*>(&b01), *reinterpret_cast<const uint32_t*>(&b23));
                        }
                        *reinterpret_cast<uint2*>(dst + quad * 8u) = wv;
                    }
                    if (c0 == 0u) {
                        const float lse2 = base - kPOffset + lg2_approx(sum);
                        if (kSplit) p.lse2[prow] = lse2;
                        else if (p.lse_nat != nullptr) p.lse_nat[(static_cast<size_t>(it.batch) * p.H + head) * p.S + row] = lse2 * 0.6931471805599453f;
                    }
                }
                continue;   // (a CTA's only unit)
            }
            float fa = 1.0f, fb = 0.0f;   // weights of the own and of the partner's half in a merge
            if (kPair && it.half == 1u) {
                join_cluster();
                ok = mbar_wait_cluster(bar_peer_data, 0u, abort_flag);
                if (!named_bar_all(kEpiBar, 128u, ok)) break;
                float2 ps;   // {l, reference} of the partner's half
                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(ps.x), "=f"(ps.y) : "r"(xch_stat) : "memory");
                ref_out = fmaxf(ref_fin, ps.y);
                fa = ex2_approx(ref_fin - ref_out);
                fb = ex2_approx(ps.y - ref_out);
                l = l * fa + ps.x * fb;
            }
            const float fin = vd / l;
            const uint32_t row = it.row0 + (r >> pack_shift), head = it.head + (r & ((1u << pack_shift) - 1u));
            if (tracing) {
                p.trace[32768 + r] = l;
                p.trace[32768 + 128 + r] = ref_out;
            }
            const bool half_out = !kSplit || kFused || (p.flags & kFlagF32Partials) == 0u;   // 16-bit rows (bf16 output, f16 partial) or f32 partial rows
            if (half_out) {
                // bf16 output, or the split kernel's f16 partial (the reference's partial format, block3.rs:291-356): four 32-column
                // chunks, all staged before the stores go out; O is free after the last read
                // Two chunks are in flight at a time: the read-out of O, which the next item's first P V waits for (o_free), then takes two
                // tensor-memory round trips and the conversion of two chunks instead of four and three (this warpgroup only gets an
                // instruction issued every few dozen clocks while the softmax warps of its scheduler run, so what stands between o_full
                // and o_free is counted in instructions)
                auto process = [&](int c, uint32_t (&o)[32]) {
                    if (dumping) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) p.trace[16384 + r * 128 + 32 * c + e] = __uint_as_float(o[e]);
                    }
                    if (kPair && it.half == 1u) {
#pragma unroll
                        for (int q4 = 0; q4 < 8; ++q4) {
                            float4 pb;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(pb.x), "=f"(pb.y), "=f"(pb.z), "=f"(pb.w)
                                         : "r"(xch_row + xch_off(c, q4)) : "memory");
                            o[4 * q4] = __float_as_uint(__uint_as_float(o[4 * q4]) * fa + pb.x * fb);
                            o[4 * q4 + 1] = __float_as_uint(__uint_as_float(o[4 * q4 + 1]) * fa + pb.y * fb);
                            o[4 * q4 + 2] = __float_as_uint(__uint_as_float(o[4 * q4 + 2]) * fa + pb.z * fb);
                            o[4 * q4 + 3] = __float_as_uint(__uint_as_float(o[4 * q4 + 3]) * fa + pb.w * fb);
                        }
                    }
                    const uint32_t tile_base = stg + (static_cast<uint32_t>(c) >> 1) * 16384u + r * 128u;
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {   // 8 columns = 16 bytes of bf16 per store
                        uint32_t wv[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            mul2(o[8 * q4 + 2 * e], o[8 * q4 + 2 * e + 1], fin);
                            const float a = __uint_as_float(o[8 * q4 + 2 * e]), b = __uint_as_float(o[8 * q4 + 2 * e + 1]);
                            if (kSplit) {
                                asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(wv[e]) : "f"(b), "f"(a));
                            } else {
                                const __nv_bfloat162 b2 = __floats2bfloat162_rn(a, b);
                                wv[e] = *reinterpret_cast<const uint32_t*>(&b2);
                            }
                        }
                        const uint32_t chunk = static_cast<uint32_t>((c & 1) * 4 + q4);
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(tile_base + ((chunk ^ (r & 7u)) << 4)),
                                     "r"(wv[0]), "r"(wv[1]), "r"(wv[2]), "r"(wv[3]) : "memory");
                    }
                };
                uint32_t oa[32], ob[32];
                tmem_ld32(t_o, oa);
                tmem_ld32(t_o + 32, ob);
                tmem_wait_ld();
                process(0, oa);
                tmem_ld32(t_o + 64, oa);
                process(1, ob);
                tmem_ld32(t_o + 96, ob);
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive(bar_o_free);   // O and L are out: the next item's first P V may overwrite them
                stamp(ep_trace, 3, 24 + static_cast<int>(n), 5);
                process(2, oa);
                process(3, ob);
                fence_proxy_async_smem();
                named_bar_sync(kEpiBar, 128u);
                if (issuer) {
                    if (kSplit) {
                        // with a routing plan the rows go to the GPU that combines them (its receive slot of this GPU), else to this launch's own partial buffer
                        const CUtensorMap* omap = &tm_o;
                        int o_row = static_cast<int>(it.row0), o_split = static_cast<int>(it.split);
                        if (!kFused && p.peer != nullptr) {
                            const uint32_t dest = it.row0 / p.peer->dest_rows;
                            omap = &p.peer->maps[dest];
                            o_row = static_cast<int>(it.row0 - dest * p.peer->dest_rows);
                            o_split = static_cast<int>(p.peer->rank);
                        }
                        tma_store_5d(omap, stg, 0, static_cast<int>(it.head), o_row, static_cast<int>(it.batch), o_split);
                        tma_store_5d(omap, stg + 16384u, 64, static_cast<int>(it.head), o_row, static_cast<int>(it.batch), o_split);
                    } else {
                        tma_store_4d(&tm_o, stg, 0, static_cast<int>(it.head), static_cast<int>(it.row0), static_cast<int>(it.batch));
                        tma_store_4d(&tm_o, stg + 16384u, 64, static_cast<int>(it.head), static_cast<int>(it.row0), static_cast<int>(it.batch));
                    }
                    bulk_commit_group();
                }
            } else {
                // f32 partial: four pieces of 32 columns (128 bytes per row), alternating between the two staging tiles; a tile is written
                // again once the store that last used it has read it out. With a routing plan the rows go to the GPU that combines them
                // (its receive slot of this GPU), else to this launch's own partial buffer.
                const CUtensorMap* omap = &tm_o;
                int o_row = static_cast<int>(it.row0), o_split = static_cast<int>(it.split);
                if (kSplit && p.peer != nullptr) {
                    const uint32_t dest = it.row0 / p.peer->dest_rows;
                    omap = &p.peer->maps[dest];
                    o_row = static_cast<int>(it.row0 - dest * p.peer->dest_rows);
                    o_split = static_cast<int>(p.peer->rank);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t o[32];
                    tmem_ld32(t_o + 32 * c, o);
                    tmem_wait_ld();
                    if (c == 3) {
                        tc_fence_before_sync();
                        mbar_arrive(bar_o_free);
                        stamp(ep_trace, 3, 24 + static_cast<int>(n), 5);
                    }
                    if (kPair && it.half == 1u) {
#pragma unroll
                        for (int q4 = 0; q4 < 8; ++q4) {
                            float4 pb;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(pb.x), "=f"(pb.y), "=f"(pb.z), "=f"(pb.w)
                                         : "r"(xch_row + xch_off(c, q4)) : "memory");
                            o[4 * q4] = __float_as_uint(__uint_as_float(o[4 * q4]) * fa + pb.x * fb);
                            o[4 * q4 + 1] = __float_as_uint(__uint_as_float(o[4 * q4 + 1]) * fa + pb.y * fb);
                            o[4 * q4 + 2] = __float_as_uint(__uint_as_float(o[4 * q4 + 2]) * fa + pb.z * fb);
                            o[4 * q4 + 3] = __float_as_uint(__uint_as_float(o[4 * q4 + 3]) * fa + pb.w * fb);
                        }
                    }
                    if (c >= 2) {   // the store of piece c - 2 (all but the newest group) must have read its tile out
                        if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                        named_bar_sync(kEpiBar, 128u);
                    }
                    const uint32_t tile_base = stg + static_cast<uint32_t>(c & 1) * 16384u + r * 128u;
#pragma unroll
                    for (int q4 = 0; q4 < 8; ++q4) {
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(tile_base + ((static_cast<uint32_t>(q4) ^ (r & 7u)) << 4)),
                                     "f"(__uint_as_float(o[4 * q4]) * fin), "f"(__uint_as_float(o[4 * q4 + 1]) * fin),
                                     "f"(__uint_as_float(o[4 * q4 + 2]) * fin), "f"(__uint_as_float(o[4 * q4 + 3]) * fin) : "memory");
                    }
                    fence_proxy_async_smem();
                    named_bar_sync(kEpiBar, 128u);
                    if (issuer) {
                        tma_store_5d(omap, stg + static_cast<uint32_t>(c & 1) * 16384u, 32 * c, static_cast<int>(it.head), o_row, static_cast<int>(it.batch), o_split);
                        bulk_commit_group();
                    }
                }
            }
            if (row < p.S && want_fin) {   // rows past the sequence are computed on clamped scales and not stored (block3.rs:194)
                const float lse2 = ref_out - kPOffset + lg2_approx(l);   // log2 of sum_j 2^(s_j)
                if (kSplit && !kFused && p.peer != nullptr) {
                    const uint32_t dest = it.row0 / p.peer->dest_rows, n_rows = p.peer->dest_rows * p.H;
                    p.peer->lse[dest][static_cast<size_t>(p.peer->rank) * n_rows + static_cast<size_t>(row - dest * p.peer->dest_rows) * p.H + head] = lse2;
                } else if (kSplit) {
                    const size_t prow = static_cast<size_t>(it.split) * p.rows_total + (static_cast<size_t>(it.batch) * p.S + row) * p.H + head;
                    p.lse2[prow] = lse2;
                } else if (p.lse_nat != nullptr) {
                    p.lse_nat[(static_cast<size_t>(it.batch) * p.H + head) * p.S + row] = lse2 * 0.6931471805599453f;
                }
            }
            if (kFused) {
                // Fused merge (the reference's last-arriver combine, tests/gpu/ref_host.cpp:489-497, docs/last-arriver-memory-model.md): every
                // CTA that has stored a partial of this 128-row block counts itself in; the one that completes the count merges the block's
                // `splits` partials into the bf16 output, so no combine kernel follows.
                // Writer side: the bulk stores of the partial are performed, every thread's log-sum-exp store is fenced, then one
                // device-scope atomic publishes both. Reader side: the atomic, a fence, copies and loads that bypass L1.
                volatile uint32_t* last_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + SmemLayout::last_flag);
                if (issuer) bulk_wait_group_done0();
                __threadfence();
                named_bar_sync(kEpiBar, 128u);
                if (issuer) {
                    uint32_t* cnt = p.fused_counters + (static_cast<size_t>(it.batch) * p.H + it.head) * p.n_qtiles + it.row0 / kRows;
                    __threadfence();
                    const uint32_t old = atomicAdd(cnt, 1u);
                    const bool last = old + 1u == p.splits;
                    if (last) *cnt = 0u;   // nobody else touches the counter any more in this launch: the next launch finds it zero
                    *last_flag = last ? 1u : 0u;
                }
                named_bar_sync(kEpiBar, 128u);
                if (*last_flag != 0u) {
                    __threadfence();
                    // The block's partial rows (256 bytes each, `splits` per output row) come in through the two staging tiles with
                    // asynchronous 16-byte copies (cp.async: no registers are tied up by loads in flight, which this warpgroup does not
                    // have), 64 rows of 256 bytes per batch (= 64 / splits output rows), two batches in flight. Piece i of a batch = the
                    // partial of split i % splits for output row i / splits, at byte 256 i of the tile; a warp's copy instruction moves two
                    // whole pieces. For the merge a warp shares an output row, 4 columns per lane.
                    const uint32_t rows_pb = 64u >> p.split_log2;
                    const uint32_t rows_valid = min(static_cast<uint32_t>(kRows), p.S - it.row0);
                    const uint32_t n_batches = (rows_valid + rows_pb - 1u) / rows_pb;
                    const size_t head_row0 = (static_cast<size_t>(it.batch) * p.S + it.row0) * p.H + it.head;   // partial row index of the block's first row
                    const uint8_t* part = static_cast<const uint8_t*>(p.ohat);
                    const uint32_t et = threadIdx.x - 32u * kFirstEpilogueWarp;   // 0 .. 127
                    auto issue = [&](uint32_t b) {   // always closes one copy group, also an empty one: two groups are in flight at any time
                        if (b < n_batches) {
                            const uint32_t first = b * rows_pb, pieces = min(rows_pb, rows_valid - first) << p.split_log2;
                            const uint32_t dst = stg + (b & 1u) * 16384u;
#pragma unroll
                            for (uint32_t i = 0; i < 8u; ++i) {
                                const uint32_t c = i * 128u + et, pc = c >> 4, ch = c & 15u;
                                if (pc < pieces) {
                                    const uint32_t row = first + (pc >> p.split_log2), sp = pc & (p.splits - 1u);
                                    const uint8_t* src = part + (static_cast<size_t>(sp) * p.rows_total + head_row0 + static_cast<size_t>(row) * p.H) * 256u + ch * 16u;
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * 16u), "l"(src) : "memory");
                                }
                            }
                        }
                        asm volatile("cp.async.commit_group;" ::: "memory");
                    };
                    issue(0u);
                    issue(1u);
                    // while the first batches fly: the block's log-sum-exps, thread r those of row r (all loads in flight at once), to shared memory
                    {
                        float lsv[8];
                        const size_t g = head_row0 + static_cast<size_t>(min(r, rows_valid - 1u)) * p.H;
#pragma unroll
                        for (uint32_t sp = 0; sp < 8u; ++sp) lsv[sp] = sp < p.splits ? __ldcg(p.lse2 + static_cast<size_t>(sp) * p.rows_total + g) : 0.0f;
                        float4* dst4 = reinterpret_cast<float4*>(smem_gen + SmemLayout::xlse + r * 32u);
                        dst4[0] = make_float4(lsv[0], lsv[1], lsv[2], lsv[3]);
                        dst4[1] = make_float4(lsv[4], lsv[5], lsv[6], lsv[7]);
                    }
                    const uint32_t tr = static_cast<uint32_t>(warp) & 3u, tc = static_cast<uint32_t>(lane);   // row within a group of 4, 8-byte column chunk
                    for (uint32_t b = 0; b < n_batches; ++b) {
                        const uint32_t first = b * rows_pb, rows_here = min(rows_pb, rows_valid - first);
                        asm volatile("cp.async.wait_group 1;" ::: "memory");   // this thread's copies of batch b have landed
                        named_bar_sync(kEpiBar, 128u);                          // everybody's have (and, the first time, the log-sum-exps are in place)
                        for (uint32_t rg = 0; rg < rows_here; rg += 4u) {
                            const uint32_t rb = rg + tr;   // row within the batch
                            if (rb < rows_here) {
                                const volatile float* ls_row = reinterpret_cast<const volatile float*>(smem_gen + SmemLayout::xlse + (first + rb) * 32u);
                                float m = -1.0e30f, den = 0.0f, acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                                const uint32_t src = stg + (b & 1u) * 16384u + ((rb << p.split_log2) << 8) + tc * 8u;
                                for (uint32_t sp = 0; sp < p.splits; ++sp) {
                                    const float ls = ls_row[sp];
                                    uint2 raw;
                                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(raw.x), "=r"(raw.y) : "r"(src + sp * 256u) : "memory");
                                    float a, w;
                                    combine_weights(m, den, ls, a, w);
                                    const float2 f01 = combine_h2_to_f2(raw.x), f23 = combine_h2_to_f2(raw.y);
                                    acc[0] = combine_accumulate(acc[0], a, w, f01.x);
                                    acc[1] = combine_accumulate(acc[1], a, w, f01.y);
                                    acc[2] = combine_accumulate(acc[2], a, w, f23.x);
                                    acc[3] = combine_accumulate(acc[3], a, w, f23.y);
                                }
                                const float rd = 1.0f / den;
                                const __nv_bfloat162 b01 = __floats2bfloat162_rn(__fmul_rn(acc[0], rd), __fmul_rn(acc[1], rd));
                                const __nv_bfloat162 b23 = __floats2bfloat162_rn(__fmul_rn(acc[2], rd), __fmul_rn(acc[3], rd));
                                uint8_t* dst = p.o + static_cast<size_t>(it.batch) * p.o_batch_stride + static_cast<size_t>(it.row0 + first + rb) * p.o_row_stride +
                                               static_cast<size_t>(it.head) * 256u + tc * 8u;
                                *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&b01), *reinterpret_cast<const uint32_t*>(&b23));
                            }
                        }
                        named_bar_sync(kEpiBar, 128u);   // everybody has read this tile out
                        issue(b + 2u);
                    }
                    asm volatile("cp.async.wait_group 0;" ::: "memory");   // (only empty groups are left)
                }
            }
            stamp(ep_trace, 3, 24 + static_cast<int>(n), 7);
        }
        if (issuer) bulk_wait_group_read0();   // the staging tiles have been read out before the CTA gives its shared memory back
    }

    // ---- teardown ----
    tc_fence_before_sync();
    __syncthreads();
    // a pair stays together to the end: the partner may still be reading this CTA's exchange area or arriving on its barrier
    if (paired) {
        join_cluster();
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
    if (threadIdx.x == 0) stamp(cta_traced ? p.trace : nullptr, 2, 30, 1);   // all roles done
    if (threadIdx.x == 0 && *abort_flag != 0u) atomicOr(p.status, 1u);
    if (warp == kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

cudaError_t launch_attention(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_o, const AttnParams& p,
                             uint32_t B, bool split, uint32_t rows_per_cta, cudaStream_t stream) {
    (void)rows_per_cta;   // both logical block heights run as 128-row CTAs
    using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const AttnParams);
    // The instantiations: [causal][recipe][trace][split] (the causal mask has no split form); behind them the variants for launches as pairs
    // of CTAs (long-sequence recipe, no mask): [trace][split]; behind those the variants with V block scales (no mask, no trace):
    // [pair][recipe][split], pairs only with the long-sequence recipe; then the split kernels with the fused merge: [V block scales][recipe];
    // then the variants that cut every item between the CTAs of a cluster: [V block scales][split], and the causal one;
    // last the variants with packed heads (the clusters' all have them): unsplit [none, causal, V block scales][recipe], split [V block scales][recipe].
#define MXA_K(split, trace, lazy, causal, pair, vbs) mxfp8_prefill_kernel<split, trace, lazy, causal, pair ? kPairs : kNoCluster, vbs>
    static const Kernel kernels[47] = {
        MXA_K(false, false, false, false, false, false), MXA_K(true, false, false, false, false, false), MXA_K(false, true, false, false, false, false),
        MXA_K(true, true, false, false, false, false),   MXA_K(false, false, true, false, false, false), MXA_K(true, false, true, false, false, false),
        MXA_K(false, true, true, false, false, false),   MXA_K(true, true, true, false, false, false),   MXA_K(false, false, false, true, false, false),
        nullptr,                                         MXA_K(false, true, false, true, false, false),  nullptr,
        MXA_K(false, false, true, true, false, false),   nullptr,                                        MXA_K(false, true, true, true, false, false),
        nullptr,
        MXA_K(false, false, true, false, true, false),   MXA_K(true, false, true, false, true, false),   MXA_K(false, true, true, false, true, false),
        MXA_K(true, true, true, false, true, false),
        MXA_K(false, false, false, false, false, true),  MXA_K(true, false, false, false, false, true),  MXA_K(false, false, true, false, false, true),
        MXA_K(true, false, true, false, false, true),    nullptr,                                        nullptr,
        MXA_K(false, false, true, false, true, true),    MXA_K(true, false, true, false, true, true),
        mxfp8_prefill_kernel<true, false, false, false, kNoCluster, false, true>, mxfp8_prefill_kernel<true, false, true, false, kNoCluster, false, true>,
        mxfp8_prefill_kernel<true, false, false, false, kNoCluster, true, true>,  mxfp8_prefill_kernel<true, false, true, false, kNoCluster, true, true>,
        mxfp8_prefill_kernel<false, false, true, false, kCutAll, false>,     mxfp8_prefill_kernel<true, false, true, false, kCutAll, false>,
        mxfp8_prefill_kernel<false, false, true, false, kCutAll, true>,      mxfp8_prefill_kernel<true, false, true, false, kCutAll, true>,
        mxfp8_prefill_kernel<false, false, true, true, kCutAll, false>,
#define MXA_PACKED(split, lazy, causal, vbs) mxfp8_prefill_kernel<split, false, lazy, causal, kNoCluster, vbs, false, true>
        MXA_PACKED(false, false, false, false), MXA_PACKED(false, true, false, false), MXA_PACKED(false, false, true, false), MXA_PACKED(false, true, true, false),
        MXA_PACKED(false, false, false, true),  MXA_PACKED(false, true, false, true),  MXA_PACKED(true, false, false, false), MXA_PACKED(true, true, false, false),
        MXA_PACKED(true, false, false, true),   MXA_PACKED(true, true, false, true)};
#undef MXA_PACKED
#undef MXA_K
    constexpr int kKernels = 47, kFirstCut = 32, kFirstPacked = 37, kCutLogs = 5;   // cut between up to 16 CTAs
    constexpr int kMaxDevices = 64;
    // per-device set-up done lazily from whichever thread launches first: plain flags would be a data race, and both steps are idempotent
    static std::atomic<bool> attr_done[kMaxDevices][kKernels];   // the shared-memory attribute is per device
    static std::atomic<int> sm_count[kMaxDevices];
    static std::atomic<int> pair_capacity[kMaxDevices][kKernels];   // -1 = not asked yet (set below on first use)
    static std::atomic<int> cut_capacity[kMaxDevices][kFirstPacked - kFirstCut][kCutLogs];   // [.][.][log2 of the cluster's CTAs]
    static std::once_flag pair_init;
    std::call_once(pair_init, [] {
        for (auto& d : cut_capacity) for (auto& k : d) for (auto& x : k) x.store(-1, std::memory_order_relaxed);
        for (auto& d : pair_capacity) for (auto& x : d) x.store(-1, std::memory_order_relaxed);
    });
    // the long-sequence recipe from 4 key tiles of the whole sequence on (crates/amdgpu-stage/src/attention/state.rs:73-77), unless the
    // caller asks for the exact one; each recipe is its own instantiation, which halves the code of the tile loop
    const bool lazy_recipe = (p.SK + kKeys - 1) / kKeys >= 4 && !(p.flags & 0x2u);
    const bool causal = (p.flags & kFlagCausal) != 0u;
    if (causal && split) return cudaErrorInvalidValue;
    const bool vbs = p.v_blockscale != nullptr;
    if (vbs && (causal || p.trace != nullptr)) return cudaErrorInvalidValue;   // V block scales: no mask, no diagnostics
    int which = vbs ? 20 + (split ? 1 : 0) + (lazy_recipe ? 2 : 0) : (split ? 1 : 0) + (p.trace != nullptr ? 2 : 0) + (lazy_recipe ? 4 : 0) + (causal ? 8 : 0);
    const bool fused = p.fused_counters != nullptr;
    if (fused && (!split || p.trace != nullptr || p.peer != nullptr || (p.flags & kFlagF32Partials) || p.splits > 8u || p.o == nullptr)) return cudaErrorInvalidValue;
    if (fused) which = 28 + (lazy_recipe ? 1 : 0) + (vbs ? 2 : 0);
    if (p.pack_shift != 0u) {
        if (p.trace != nullptr || p.peer != nullptr || fused) return cudaErrorInvalidValue;
        which = kFirstPacked + (lazy_recipe ? 1 : 0) + (split ? 6 + (vbs ? 2 : 0) : (causal ? 2 : 0) + (vbs ? 4 : 0));
    }
    const int which_pair = vbs ? 26 + (split ? 1 : 0) : 16 + (split ? 1 : 0) + (p.trace != nullptr ? 2 : 0);   // only for the long-sequence recipe without a mask
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    auto ensure_attr = [&](int k) -> cudaError_t {
        if (attr_done[dev][k].load(std::memory_order_acquire)) return cudaSuccess;
        cudaError_t ea = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernels[k]), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (ea == cudaSuccess && k >= kFirstCut && k < kFirstPacked)
            ea = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernels[k]), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);   // 16 CTAs, where they fit
        if (ea == cudaSuccess) attr_done[dev][k].store(true, std::memory_order_release);
        return ea;
    };
    e = ensure_attr(which);
    if (e != cudaSuccess) return e;
    int sms = sm_count[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        int n = 0;
        e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        sms = n > 0 ? n : 1;
        sm_count[dev].store(sms, std::memory_order_relaxed);
    }
    // Persistent launch: one CTA per SM (a CTA takes all of an SM's tensor memory and nearly all of its shared memory), each walking the
    // work units blockIdx.x, blockIdx.x + gridDim.x, ...
    AttnParams q = p;
    const uint32_t seq_rows = kRows >> p.pack_shift;   // sequence rows of an item
    q.n_qtiles = (p.S + seq_rows - 1) / seq_rows;
    const unsigned long long items = 1ull * q.n_qtiles * (p.H >> p.pack_shift) * B * (split ? p.splits : 1u);
    if (items == 0 || items > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    q.n_items = static_cast<uint32_t>(items);
    q.n_work = q.n_items;
    q.tail_base = q.n_items;
    q.tail_split = 0u;
    uint32_t ctas = q.n_items < static_cast<uint32_t>(sms) ? q.n_items : static_cast<uint32_t>(sms);
    // The last round. n_items = rounds * grid + tail: when the tail fills at most half of the grid, its items would keep a few CTAs busy
    // for a whole item while the rest idle. They are then cut in two key ranges each, the grid is launched as clusters of two CTAs, and
    // each pair merges its two halves through distributed shared memory (no workspace). Long-sequence recipe only (integer references
    // merge exactly), no causal mask (its items differ in length and are balanced by their order), and only for items of at least
    // kMinTilesForPairs key tiles: a launch as pairs and the merge cost about 7-9 us (measured), which half an item has to outweigh.
    const uint32_t ntiles_total = (p.SK + kKeys - 1) / kKeys;
    uint32_t min_tiles = ntiles_total;
    if (split) {
        const uint32_t tps = (ntiles_total + p.splits - 1) / p.splits;
        min_tiles = ntiles_total - (p.splits - 1u) * tps;   // the last split's share
    }
    const uint32_t even_sms = static_cast<uint32_t>(sms) & ~1u;
    constexpr uint32_t kMinTilesForPairs = 48u;
    // how many clusters of `cluster` CTAs of kernel k the device holds at once (asked once per device, kernel and size, and kept in `known`)
    auto clusters_that_fit = [&](int k, uint32_t cluster, std::atomic<int>& known) -> uint32_t {
        int n = known.load(std::memory_order_relaxed);
        if (n < 0) {
            cudaLaunchConfig_t probe = {};
            probe.gridDim = dim3(static_cast<uint32_t>(sms) / cluster * cluster, 1, 1);
            probe.blockDim = dim3(kThreads, 1, 1);
            probe.dynamicSmemBytes = kSmemBytes;
            cudaLaunchAttribute pa[1];
            pa[0].id = cudaLaunchAttributeClusterDimension;
            pa[0].val.clusterDim.x = cluster; pa[0].val.clusterDim.y = 1; pa[0].val.clusterDim.z = 1;
            probe.attrs = pa;
            probe.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(kernels[k]), &probe) != cudaSuccess) { n = 0; (void)cudaGetLastError(); }
            known.store(n, std::memory_order_relaxed);
        }
        return static_cast<uint32_t>(n);
    };
    uint32_t cluster_ctas = 1u;
    // Few items: each is cut between the CTAs of a cluster, as far as the machine holds the clusters at once and it is worth it. The merge stays in shared
    // memory, with f32 partials and no workspace. What it costs, in key tiles of 0.58 us (1140 clocks at 1965 MHz): the launch as clusters
    // 8 (64 items of 4 valid rows, 16 tiles: 15.2 us whole, 15.6 us as halves; 32 tiles: 24.7 and 20.3), the exchange of 128 rows another 5 (64 items of 128 rows,
    // 16 tiles: 15.8 and 18.2 us; 32 tiles: 25.5 and 23.3; 8 items, 16 tiles, in 16 parts: 13.9 and 13.3). With the first copies in the set-up both forms start earlier and
    // the rule still takes the faster one: 64 items of 128 rows, 32 tiles 24.8 whole and 21.6 as halves; of 4 rows 23.0 and 18.6; 20 items, 24 tiles 17.9 and 14.6; 8 items, 16 tiles
    // 13.2 and 12.1, 64 tiles 39.2 and 15.9. Cutting only the last of several rounds this way gained
    // 1 % at 64 tiles and lost 4 % at 16: not done.
    const bool plain = p.trace == nullptr && p.peer == nullptr && !fused && !(p.flags & (kFlagF32Partials | kFlagNoTailSplit));
    if (lazy_recipe && plain && 2u * q.n_items <= static_cast<uint32_t>(sms)) {
        uint32_t tiles = min_tiles;
        if (causal) tiles = (min(p.SK, seq_rows + (p.SK - p.S)) + kKeys - 1) / kKeys;   // the first row block's
        const int k_cut = causal ? kFirstCut + 4 : kFirstCut + (split ? 1 : 0) + (vbs ? 2 : 0);
        const uint32_t merge_tiles = 8u + 5u * min(p.S << p.pack_shift, static_cast<uint32_t>(kRows)) / kRows;
        uint32_t lg = 0, best = tiles;
        for (uint32_t l = 1; l < kCutLogs && (q.n_items << l) <= static_cast<uint32_t>(sms) && (tiles >> l) > 0u; ++l) {
            const uint32_t cost = ((tiles + (1u << l) - 1u) >> l) + merge_tiles;
            if (cost < best) { best = cost; lg = l; }
        }
        if (lg > 0) {
            e = ensure_attr(k_cut);
            if (e != cudaSuccess) return e;
        }
        while (lg > 0 && clusters_that_fit(k_cut, 1u << lg, cut_capacity[dev][k_cut - kFirstCut][lg]) < q.n_items) --lg;
        if (lg > 0) {
            q.cut_log2 = lg;
            cluster_ctas = 1u << lg;
            q.n_work = q.n_items << lg;
            q.tail_base = q.n_work;
            ctas = q.n_work;
            which = k_cut;
        }
    }
    if (cluster_ctas == 1u && lazy_recipe && !causal && !fused && min_tiles >= kMinTilesForPairs && even_sms >= 2u && !(p.flags & kFlagNoTailSplit)) {
        const uint32_t rounds = q.n_items / even_sms, tail = q.n_items - rounds * even_sms;
        if (tail > 0u && 2u * tail <= even_sms) {
            const uint32_t grid = rounds > 0u ? even_sms : 2u * tail;
            e = ensure_attr(which_pair);
            if (e != cudaSuccess) return e;
            if (clusters_that_fit(which_pair, 2u, pair_capacity[dev][which_pair]) * 2u >= grid) {
                q.tail_split = 1u;
                q.tail_base = rounds * even_sms;
                q.n_work = q.tail_base + 2u * tail;
                ctas = grid;
                which = which_pair;
                cluster_ctas = 2u;
            }
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // overlap this grid's launch and set-up with the tail of the grid before it
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster_ctas > 1u) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster_ctas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, kernels[which], tm_q, tm_k, tm_v, tm_o, q);
}

}  // namespace b200mx
