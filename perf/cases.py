"""Performance cases of the MXFP8 attention path: what a user of this package has it do, through its public Python entry points.

A case is one of three kinds of pass:

  attend           `fmha_fwd_mxfp8` on e4m3 Q, K, V with E8M0 scales that are already on the GPU
  quantize         `quantize_qk` on Q and K and `quantize_v` on V: bf16 activations to the operands of `attend`
  quantize_attend  both, as a layer that gets bf16 activations calls them

Keys of a case: B, H, HK, S, SK (batch, query heads, KV heads, query rows, keys); for the attending kinds also `path` and `splits` (as the entry
point takes them; splits 0: not given), `causal`, `lse` (natural log-sum-exps wanted too) and `v_blocks` (V with one E8M0 per 32 keys and column
instead of one descale per tensor).

Inputs are seeded normal tensors quantised by the package's own quantisers; the queries of each head carry a gain between a half and three,
so that the softmax rows range from flat to peaked as the heads of a trained model's do.
"""
import math

import torch

from amdgpu_rustdsl_b200 import Q_PRESCALE, fmha_fwd_mxfp8, quantize_qk, quantize_v

D = 128
ATTEND = {"path": "auto", "splits": 0, "causal": False, "lse": False, "v_blocks": False}


def _attend(name, B, H, HK, S, SK, **options):
    return {"name": name, "kind": "attend", "B": B, "H": H, "HK": HK, "S": S, "SK": SK, **ATTEND, **options}


def listed():
    return [
        # the smallest call: one short prompt on two heads (first shape of the benchmark), where launches and host time are all there is
        _attend("tiny_s256", 1, 2, 2, 256, 256),
        # one new token for each of 16 sequences with a 4096-key cache, grouped heads: a decode step
        _attend("decode_b16_sk4096", 16, 32, 8, 1, 4096),
        # a batch of two prompts of odd lengths with grouped heads; the log-sum-exps are what a caller merging attention over parts asks for
        _attend("ragged_gqa_lse", 2, 16, 4, 1000, 1337, lse=True),
        # a single 2048-token prompt: too few row blocks for the machine, the dispatch takes the key split
        _attend("prefill_b1_s2048", 1, 8, 8, 2048, 2048),
        # the headline shape of the benchmark
        _attend("prefill_b4_s2048", 4, 8, 8, 2048, 2048),
        # the same with one scale per 32 keys on V
        _attend("prefill_b4_s2048_vblocks", 4, 8, 8, 2048, 2048, v_blocks=True),
        # prefill of a language model's layer: causal, grouped heads
        _attend("causal_gqa_s4096", 1, 32, 8, 4096, 4096, causal=True),
        # a 512-token chunk of a long prompt against the cache of what came before
        _attend("chunk_s512_sk16384", 1, 16, 4, 512, 16384),
        # long context with the split forced to eight ways (third shape of the benchmark)
        _attend("split8_s8192", 1, 8, 8, 8192, 8192, path="kvsplit", splits=8),
        # the largest shape of the benchmark on one GPU
        _attend("prefill_b16_h64_s4096", 16, 64, 64, 4096, 4096),
        # bf16 activations of a large batch to the path's operands
        {"name": "quantize_b8_s4096", "kind": "quantize", "B": 8, "H": 32, "HK": 8, "S": 4096, "SK": 4096},
        # a short prompt from bf16 activations to bf16 output: a chain of small launches
        {"name": "quantize_attend_s1000", "kind": "quantize_attend", "B": 1, "H": 8, "HK": 2, "S": 1000, "SK": 1000, **ATTEND},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _pairs(case):
    """(query, key) pairs the mask leaves, per (batch, head)."""
    S, SK = case["S"], case["SK"]
    return S * (SK - S) + S * (S + 1) // 2 if case.get("causal") else S * SK


def draw(rng):
    """A case of the same ranges: 1 to 16 sequences, 1 to 64 heads in groups of 1 to 8, 1 to 8192 query rows, 1 to 32768 keys, any option that
    the entry point takes at these sizes; no more work than the largest listed case."""
    while True:
        kind = rng.choice(["attend"] * 8 + ["quantize"] * 2 + ["quantize_attend"] * 2)
        gqa = rng.choice([1, 1, 2, 4, 8])
        case = {"kind": kind, "B": _log_uniform(rng, 1, 16), "HK": _log_uniform(rng, 1, 64 // gqa)}
        case["H"] = case["HK"] * gqa
        use = rng.choice(["prefill", "prefill", "prefill", "decode", "chunk"])
        if use == "prefill":      # self-attention of whole prompts
            case["S"] = case["SK"] = _log_uniform(rng, 64, 8192)
        elif use == "decode":     # one or a few new tokens over a cache
            case["S"], case["SK"] = _log_uniform(rng, 1, 16), _log_uniform(rng, 256, 32768)
        else:                     # part of a prompt over a cache, or cross-attention
            case["S"], case["SK"] = _log_uniform(rng, 32, 2048), _log_uniform(rng, 256, 32768)
        if rng.random() < 0.3:    # round sizes are common too
            case["S"], case["SK"] = (x if x < 64 else -(-x // 64) * 64 for x in (case["S"], case["SK"]))
        if kind != "quantize":
            case.update(ATTEND)
            option = rng.choice(["none", "none", "none", "causal", "lse", "v_blocks", "kvsplit"])
            if option == "causal":
                case["causal"] = True
                case["SK"] = max(case["SK"], case["S"])
            elif option == "lse":
                # the split path has no log-sum-exp output: ask for one of the unsplit kernels
                case["lse"], case["path"] = True, "vs128"
            elif option == "v_blocks" and kind == "attend":
                case["v_blocks"] = True
            elif option == "kvsplit":
                splits, tiles = rng.choice([2, 4, 8]), -(-case["SK"] // 128)
                if (splits - 1) * -(-tiles // splits) < tiles:   # every split needs a tile of keys
                    case["path"], case["splits"] = "kvsplit", splits
        rows, keys = case["B"] * case["S"] * case["H"], case["B"] * case["SK"] * case["HK"]
        if rows <= 1 << 21 and keys <= 1 << 21 and (kind == "quantize" or 4 * case["B"] * case["H"] * _pairs(case) * D <= 4e12):
            return case


def _normal(g, shape, gain=None):
    """bf16 normal samples, made one batch element at a time to keep the f32 samples small."""
    x = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    for b in range(shape[0]):
        y = torch.randn(shape[1:], generator=g, device="cuda")
        x[b] = y if gain is None else y * gain
    return x


def _v_block_scaled(v):
    """V [B, SK, HK, 128] to e4m3 bytes and E8M0 [B, ceil(SK / 32), HK, 128]: one scale per 32 keys and column."""
    B, SK, HK, _ = v.shape
    blocks = -(-SK // 32)
    x = torch.nn.functional.pad(v.float(), (0, 0, 0, 0, 0, blocks * 32 - SK)).view(B, blocks, 32, HK, D)
    exponent = torch.frexp(x.abs().amax(dim=2)).exponent - 1 - 8
    scale = (exponent + 127).clamp(1, 254)
    x = torch.ldexp(x, (127 - scale).unsqueeze(2)).clamp(-448, 448).to(torch.float8_e4m3fn)
    return x.view(torch.uint8).reshape(B, blocks * 32, HK, D)[:, :SK].contiguous(), scale.to(torch.uint8).contiguous()


def prepare(case, seed):
    B, H, HK, S, SK = (case[x] for x in ("B", "H", "HK", "S", "SK"))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    gain = torch.exp2(torch.rand(H, 1, generator=g, device="cuda") * 2.6 - 1.0)
    q, k, v = _normal(g, (B, S, H, D), gain), _normal(g, (B, SK, HK, D)), _normal(g, (B, SK, HK, D))
    s = {"case": case}
    # operand buffers, with the zeroed slack behind the scales that the entry point's contract asks for
    s["q8"], s["k8"], s["v8"] = (torch.empty(x.shape, dtype=torch.uint8, device="cuda") for x in (q, k, v))
    s["qs"] = torch.zeros(B * S * H * 4 + 512 * H * 4, dtype=torch.uint8, device="cuda")
    s["ks"] = torch.zeros(B * SK * HK * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda")
    s["vs"] = torch.zeros(1024, dtype=torch.float32, device="cuda")
    s["v_descale"] = s["vs"][:1]   # the rest of the buffer is the quantiser's scratch and the contract's padding
    if case["kind"] != "quantize":
        s["out"] = torch.empty((B, S, H, D), dtype=torch.bfloat16, device="cuda")
        s["options"] = {"path": case["path"], "splits": case["splits"] or None, "causal": case["causal"]}
        if case["lse"]:
            s["options"]["lse"] = torch.empty((B, H, S), dtype=torch.float32, device="cuda")
    if case["kind"] == "attend":
        quantize_qk(q, s["q8"], s["qs"], mul=Q_PRESCALE)
        quantize_qk(k, s["k8"], s["ks"])
        if case["v_blocks"]:
            s["v8"], s["options"]["v_blockscale"] = _v_block_scaled(v)
        else:
            quantize_v(v, s["v8"], s["vs"])
    else:
        s["q"], s["k"], s["v"] = q, k, v
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind != "attend":
        quantize_qk(s["q"], s["q8"], s["qs"], mul=Q_PRESCALE)
        quantize_qk(s["k"], s["k8"], s["ks"])
        quantize_v(s["v"], s["v8"], s["vs"])
        operands = [s["q8"], s["qs"], s["k8"], s["ks"], s["v8"], s["v_descale"]]
        if kind == "quantize":
            return operands
    fmha_fwd_mxfp8(s["q8"], s["k8"], s["v8"], s["qs"], s["ks"], s["vs"], s["out"], **s["options"])
    outputs = [s["out"], s["options"]["lse"]] if s["case"]["lse"] else [s["out"]]
    return outputs if kind == "attend" else outputs + operands


def work(case):
    B, H, HK, S, SK = (case[x] for x in ("B", "H", "HK", "S", "SK"))
    rows, keys = B * S * H, B * SK * HK
    operands = (rows + keys) * (D + 4) + keys * D   # e4m3 Q, K, V and the E8M0 bytes of Q and K
    n_bytes = n_flops = 0
    if case["kind"] != "attend":
        n_bytes += (rows + 2 * keys) * 2 * D + operands   # bf16 read once, the operands written once
        n_flops += 3 * (rows + 2 * keys) * D              # magnitude for the scale, scaling, rounding
    if case["kind"] != "quantize":
        n_bytes += rows * 2 * D + (operands if case["kind"] == "attend" else 0)
        n_bytes += rows * 4 if case["lse"] else 0
        n_bytes += B * -(-SK // 32) * HK * D if case["v_blocks"] else 0
        n_flops += 4 * B * H * _pairs(case) * D
    return {"bytes": n_bytes, "flops": n_flops}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"
    # P is e4m3 in front of P V: rounding to three mantissa bits is off by 2^-4 at most, about 0.026 in the root mean square, and with keys of
    # random sign the error of a row's output is that share of its norm; two implementations that scale P differently round differently. bf16 O
    # adds 2^-9. Single elements: a few dozen keys carry a peaked row, an element is then off by a few such steps of one key's weight.
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}
