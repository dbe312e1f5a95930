"""Query heads of a KV head packed into one row block, and row blocks cut between the CTAs of a cluster: against the same call with every head on
its own K and V (nothing to pack) and with FMHA_MXFP8_FLAG_NO_TAIL_SPLIT (nothing cut), which the other GPU tests hold against the fp64 oracle."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _inputs(B, H, HK, S, SK, seed=3):
    from amdgpu_rustdsl_b200 import Q_PRESCALE, quantize_qk, quantize_v
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16) for shape in ((B, S, H, 128), (B, SK, HK, 128), (B, SK, HK, 128)))
    q *= torch.linspace(0.5, 3.0, H, device="cuda")[:, None].to(torch.bfloat16)
    q8, k8, v8 = (torch.empty(x.shape, dtype=torch.uint8, device="cuda") for x in (q, k, v))
    qs = torch.zeros(B * S * H * 4 + 512 * H * 4, dtype=torch.uint8, device="cuda")
    ks = torch.zeros(B * SK * HK * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda")
    vs = torch.zeros(1024, dtype=torch.float32, device="cuda")
    quantize_qk(q, q8, qs, mul=Q_PRESCALE)
    quantize_qk(k, k8, ks)
    quantize_v(v, v8, vs)
    vb = torch.randint(120, 128, (B, -(-SK // 32), HK, 128), generator=g, device="cuda", dtype=torch.uint8)
    return q8, k8, v8, qs, ks, vs, vb


def _run(d, path, splits, causal, vblocks, flags):
    from amdgpu_rustdsl_b200 import device_status, fmha_fwd_mxfp8
    q, k, v, qs, ks, vs, vb = d
    B, S, H, _ = q.shape
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    lse = torch.full((B, H, S), float("nan"), device="cuda") if path != "kvsplit" else None
    fmha_fwd_mxfp8(q, k, v, qs, ks, vs, out, path=path, splits=splits, causal=causal, flags=flags, lse=lse, v_blockscale=vb if vblocks else None)
    torch.cuda.synchronize()
    assert device_status() == 0
    return out, lse


def _ungrouped(d, g):
    q, k, v, qs, ks, vs, vb = d
    B, SK, HK, _ = k.shape
    spread = lambda x, dim: x.repeat_interleave(g, dim=dim).contiguous()   # noqa: E731
    scales = spread(ks[: B * SK * HK * 4].view(B, SK, HK, 4), 2).flatten()
    ks2 = torch.cat([scales, torch.zeros(640 * HK * g * 4, dtype=torch.uint8, device="cuda")])
    return q, spread(k, 2), spread(v, 2), qs, ks2, vs, spread(vb, 2)


def _exact(d, causal, vblocks):
    q, k, v, qs, ks, vs, vb = d
    (B, S, H, _), (_, SK, HK, _) = q.shape, k.shape
    e4m3 = lambda x: x.view(torch.float8_e4m3fn).double()   # noqa: E731
    scale = lambda e: torch.exp2(e.double() - 127.0)   # noqa: E731
    qd = e4m3(q) * scale(qs[: B * S * H * 4].view(B, S, H, 4)).repeat_interleave(32, dim=3)
    kd = e4m3(k) * scale(ks[: B * SK * HK * 4].view(B, SK, HK, 4)).repeat_interleave(32, dim=3)
    vd = e4m3(v) * (scale(vb).repeat_interleave(32, dim=1)[:, :SK] if vblocks else vs[0].double())
    kd, vd = (x.repeat_interleave(H // HK, dim=2) for x in (kd, vd))
    s = torch.einsum("bihd,bjhd->bhij", qd, kd) * math.log(2.0)
    if causal:
        i, j = torch.arange(S, device="cuda")[:, None], torch.arange(SK, device="cuda")[None]
        s.masked_fill_(j >= i + SK - S + 1, -math.inf)
    return torch.einsum("bhij,bjhd->bihd", s.softmax(-1), vd), s.logsumexp(-1)


@pytest.mark.parametrize("shape", [(2, 8, 2, 1, 700), (1, 16, 1, 3, 300), (3, 4, 2, 65, 1337), (1, 32, 2, 9, 640), (2, 8, 1, 130, 512), (1, 8, 2, 33, 129)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("option", ["plain", "causal", "vblocks", "kvsplit"])
def test_packed_heads_give_the_bytes_of_separate_heads(shape, option):
    from amdgpu_rustdsl_b200 import _abi
    B, H, HK, S, SK = shape
    d = _inputs(*shape)
    path, splits = ("kvsplit", 2) if option == "kvsplit" else ("vs128", None)
    got, want = (_run(x, path, splits, option == "causal", option == "vblocks", _abi.FLAG_NO_TAIL_SPLIT) for x in (d, _ungrouped(d, H // HK)))
    assert torch.equal(got[0].view(torch.int16), want[0].view(torch.int16))
    assert got[1] is None or torch.equal(got[1].view(torch.int32), want[1].view(torch.int32))


# cut between 2, 4, 8 and 16 CTAs (as far as the device holds such clusters), with ragged ends, one row, full row blocks and rows past the sequence
@pytest.mark.parametrize("shape", [(1, 8, 1, 1, 512), (1, 1, 1, 1, 32768), (2, 8, 2, 5, 8191), (1, 4, 4, 300, 4100), (1, 2, 2, 128, 16384), (8, 8, 1, 16, 3000), (1, 16, 4, 512, 2049)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("option", ["plain", "causal", "vblocks", "kvsplit"])
def test_items_cut_between_ctas_agree_with_whole_items(shape, option):
    from amdgpu_rustdsl_b200 import _abi
    d = _inputs(*shape, seed=5)
    path, splits = ("kvsplit", 2) if option == "kvsplit" else ("vs128", None)
    (got, got_lse), (want, want_lse) = (_run(d, path, splits, option == "causal", option == "vblocks", f) for f in (0, _abi.FLAG_NO_TAIL_SPLIT))
    ref, ref_lse = _exact(d, option == "causal", option == "vblocks")
    err = [(x.double() - ref).norm().item() for x in (got, want)]
    # A part's references start from its own keys, where the whole item's start from its first: on average no weight of P is further below its reference, and
    # measured the parts' error is 0.64 to 1.00 of the whole items'. A single row's reference may sit up to 3.5 binades higher in a part than in the
    # item, and its keys far below it then round more coarsely: the allowance for that is 0.3 of a row's error, which averages out over B H S rows. The other
    # share is the rounding of the bf16 output
    rows = shape[0] * shape[1] * shape[3]
    assert err[0] <= (1 + 0.3 / math.sqrt(rows)) * err[1] + 2.0 ** -9 * ref.norm().item(), err
    # a weight is off by 2^-4 from e4m3 rounding and 0.062 from the linear mantissa at most, in the sum as in the product
    vmax = 448.0 if option == "vblocks" else 448.0 * d[5][0].item()   # (block scales up to 2^0)
    assert (got.double() - ref).abs().max().item() <= 2 * 0.125 / (1 - 0.125) * vmax
    if got_lse is not None:
        assert (got_lse.double() - ref_lse).abs().max().item() <= 0.134   # -ln(1 - 0.125)


@pytest.mark.parametrize("shape,ref_log2", [((1, 8, 8, 2048, 2048), 2), ((1, 8, 2, 1, 4096), 3), ((2, 4, 4, 1000, 2050), 2), ((1, 16, 4, 512, 16384), 0), ((1, 8, 2, 1, 32768), 0)], ids=lambda s: str(s).replace(" ", ""))
def test_a_dispatched_split_runs_as_the_faster_of_the_two_forms(shape, ref_log2):
    """The entry reports the dispatch's answer either way, and gives the bytes of the form that the rule names."""
    from amdgpu_rustdsl_b200 import _abi, fmha_fwd_mxfp8, select_path
    B, H, HK, S, SK = shape
    path, splits = select_path(B, H, S, SK)
    assert path == "kvsplit" and _abi.load().fmha_mxfp8_auto_unsplit(B, H, HK, S, SK, splits) == ref_log2
    q, k, v, qs, ks, vs, _ = d = _inputs(*shape)
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert fmha_fwd_mxfp8(q, k, v, qs, ks, vs, out) == (path, splits)
    want, _ = _run(d, "vs128" if ref_log2 else path, None if ref_log2 else splits, False, False, ref_log2 << _abi.FLAG_REF_TILES_SHIFT)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    # No further from 64 bits than the split itself: the same weights of P but for a shorter run, and f32 partials for f16 ones. The share is for errors that
    # cancel in one of the two; 2^-9 is the rounding of the bf16 output
    ref, _ = _exact(d, False, False)
    split, _ = _run(d, path, splits, False, False, 0)
    err = [(x.double() - ref).norm().item() for x in (out, split)]
    assert err[0] <= 1.03 * err[1] + 2.0 ** -9 * ref.norm().item(), err


# keys of which 32-key blocks are masked by a bias column: the first block, the first tile, the second, the last block, two of three
MASKS = {"block0": lambda b, n: b == 0, "tile0": lambda b, n: b < 4, "tile1": lambda b, n: (b >= 4) & (b < 8), "last": lambda b, n: b == n - 1, "most": lambda b, n: b % 3 != 1}


@pytest.mark.parametrize("pattern", MASKS)
@pytest.mark.parametrize("lowest", [False, True])   # scores of -inf, or of about -2^125
@pytest.mark.parametrize("shape,option", [((1, 2, 2, 200, 1337), "plain"), ((2, 8, 2, 3, 4096), "plain"), ((1, 2, 2, 700, 1000), "causal"), ((1, 2, 1, 256, 2100), "kvsplit"), ((1, 2, 2, 300, 8300), "vblocks")],
                         ids=lambda s: s if isinstance(s, str) else "x".join(map(str, s)))
def test_masked_blocks_of_keys_have_no_weight(pattern, lowest, shape, option):
    """A column of 448 in Q against -448 in K with a large scale takes a key out of the softmax, whichever blocks and tiles have no other keys."""
    q, k, v, qs, ks, vs, vb = d = _inputs(*shape, seed=8)
    B, H, HK, S, SK = shape
    blocks = torch.arange(SK, device="cuda") // 32
    masked = MASKS[pattern](blocks, int(blocks[-1]) + 1)
    q[..., 0] = 0x7E
    qs[: B * S * H * 4].view(B, S, H, 4)[..., 0] = 127
    k[..., 0] = 0
    k[:, masked, :, :32] = 0
    k[:, masked, :, 0] = 0xFE
    ks[: B * SK * HK * 4].view(B, SK, HK, 4)[:, masked, :, 0] = 127 + 107 if lowest else 254
    path, splits = ("kvsplit", 2) if option == "kvsplit" else ("vs128", None)
    got, got_lse = _run(d, path, splits, option == "causal", option == "vblocks", 0)
    ref, ref_lse = _exact(d, option == "causal", option == "vblocks")
    # a weight is off by 2^-4 from e4m3 rounding and 0.062 from the linear mantissa at most, in the sum as in the product
    vmax = 448.0 if option == "vblocks" else 448.0 * vs[0].item()
    assert torch.isfinite(got).all() and (got.double() - ref).abs().max().item() <= 2 * 0.125 / (1 - 0.125) * vmax
    if got_lse is not None:
        assert (got_lse.double() - ref_lse).abs().max().item() <= 0.134   # -ln(1 - 0.125)


def test_the_callers_reference_run_is_kept_on_the_default_path():
    """The REF_TILES field in the caller's flags: the default path does not put its own number over it, here (1) or in the C entry, and runs the split."""
    import ctypes as C
    from amdgpu_rustdsl_b200 import _abi, fmha_fwd_mxfp8, select_path
    shape = B, H, HK, S, SK = 1, 8, 8, 2048, 2048
    path, splits = select_path(B, H, S, SK)
    lib, flags = _abi.load(), 1 << _abi.FLAG_REF_TILES_SHIFT
    assert path == "kvsplit" and lib.fmha_mxfp8_auto_unsplit(B, H, HK, S, SK, splits) == 2
    q, k, v, qs, ks, vs, _ = d = _inputs(*shape)
    want, _ = _run(d, path, splits, False, False, flags)
    out, out_c = (torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert fmha_fwd_mxfp8(q, k, v, qs, ks, vs, out, flags=flags) == (path, splits)
    ws_o, ws_l = (torch.empty(splits * B * S * H * n, dtype=torch.uint8, device="cuda") for n in (512, 4))
    pr = _abi.Problem(B=B, H=H, HK=HK, S=S, SK=SK, q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), q_descale=qs.data_ptr(), k_descale=ks.data_ptr(), v_descale=vs.data_ptr(),
                      out=out_c.data_ptr(), q_descale_bytes=qs.numel(), k_descale_bytes=ks.numel(), v_descale_bytes=4096, ws_ohat=ws_o.data_ptr(), ws_lse=ws_l.data_ptr(),
                      ws_ohat_bytes=ws_o.numel(), ws_lse_bytes=ws_l.numel(), v_blockscale=None, flags=flags)
    err = C.create_string_buffer(256)
    assert lib.fmha_mxfp8_auto(C.byref(pr), -1, 0, None, None, None, err, 256) == 0, err.value
    torch.cuda.synchronize()
    for x in (out, out_c):
        assert torch.equal(x.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("shape", [(1, 8, 8, 2048, 2048), (1, 16, 4, 512, 16384), (1, 8, 2, 1, 32768)], ids=lambda s: "x".join(map(str, s)))
def test_the_default_path_writes_the_log_sum_exps_it_is_asked_for(shape):
    """Shapes that the dispatch splits (one that runs unsplit anyway, two that do not): the split has no such output, so an unsplit kernel runs and is reported."""
    from amdgpu_rustdsl_b200 import fmha_fwd_mxfp8, select_path
    B, H, HK, S, SK = shape
    path, splits = select_path(B, H, S, SK)
    assert path == "kvsplit"
    q, k, v, qs, ks, vs, _ = d = _inputs(*shape)
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    lse = torch.full((B, H, S), float("nan"), device="cuda")
    assert fmha_fwd_mxfp8(q, k, v, qs, ks, vs, out, lse=lse) == ("vs128", 0)
    ref, ref_lse = _exact(d, False, False)
    assert (lse.double() - ref_lse).abs().max().item() <= 0.134   # -ln(1 - 0.125): weights off by 0.125 at most
    # no further from 64 bits than the split (the same weights of P but for a shorter run; the allowances of the test above)
    split, _ = _run(d, path, splits, False, False, 0)
    err = [(x.double() - ref).norm().item() for x in (out, split)]
    assert err[0] <= 1.03 * err[1] + 2.0 ** -9 * ref.norm().item(), err
