"""The quantisers in front of the path. CPU: the oracle's restatement of the harness's host rule (tests/gpu/ref_host.cpp:239-258) turns the
`normal` generator's unquantised samples into exactly the generator's bytes. GPU: the device quantisers, through the C ABI, equal that
restatement bit for bit, edge cases included, and their output drives the attention kernels through the usual gate."""
import numpy as np
import pytest


@pytest.mark.parametrize("shape", [(1, 2, 256, 512, 2), (2, 4, 77, 130, 1), (1, 8, 64, 64, 8)], ids=lambda s: "B%dH%dS%dSK%dHK%d" % s)
def test_oracle_quantiser_reproduces_the_generator_bytes(oracle, shape):
    B, H, S, SK, HK = shape
    inp = oracle.generate("normal", B, H, S, SK, HK)
    q, k, v = oracle.generate_raw_normal(B, H, S, SK, HK)
    qb, qs = oracle.quantize_rows(q)          # the generator folds the softmax scale into its Q samples before quantising
    kb, ks = oracle.quantize_rows(k)
    vb, vd = oracle.quantize_tensor(v)
    assert np.array_equal(qb.reshape(inp.q.shape), inp.q) and np.array_equal(qs.ravel(), inp.qs[: qs.size])
    assert np.array_equal(kb.reshape(inp.k.shape), inp.k) and np.array_equal(ks.ravel(), inp.ks[: ks.size])
    assert np.array_equal(vb.reshape(inp.v.shape), inp.v) and vd == np.float32(inp.vdescale)


def test_oracle_quantiser_edge_cases(oracle):
    x = np.zeros((4, 128), np.float32)
    x[1, :32] = 448.0          # amax = 448 = 1.75 * 2^8: scale 2^0, top element exactly representable
    x[1, 32:64] = 449.0        # scale still 2^0: saturates to 448
    x[2, 0] = 2.0 ** -140      # subnormal maximum: scale clamps at E8M0 0
    x[3, :] = np.linspace(-3, 3, 128, dtype=np.float32)
    out, sc = oracle.quantize_rows(x)
    assert sc[0].tolist() == [0, 0, 0, 0] and not out[0].any()
    assert sc[1, 0] == 127 and out[1, 0] == 126 and sc[1, 1] == 127 and out[1, 32] == 126
    assert sc[2, 0] == 0
    tab = oracle.e4m3_table()
    deq = tab[out[3]].reshape(4, 32) * (2.0 ** (sc[3].astype(np.float64) - 127))[:, None]
    assert np.abs(deq.ravel() - x[3]).max() <= 2.0 ** -4 * 3.0      # e4m3 has 3 mantissa bits: half an ulp of 2^-3 relative


@pytest.mark.gpu
def test_device_quantisers_equal_the_oracle_bit_for_bit(oracle):
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import Q_PRESCALE, quantize_qk, quantize_v
    rng = np.random.default_rng(7)
    for rows in (1, 3, 16, 1000, 65536 + 5):
        x = (rng.standard_normal((rows, 128)) * np.exp2(rng.integers(-12, 12, (rows, 1)))).astype(np.float32)
        x[0, :32] = 0.0
        if rows > 2:
            x[1, 5] = 3.0e38
            x[2, :] = 2.0 ** -130
        xb = torch.from_numpy(x).to(torch.bfloat16).cuda()
        xf = xb.float().cpu().numpy()                      # the bf16 values the device sees
        for mul in (1.0, Q_PRESCALE):
            out = torch.full((rows, 128), 0xAA, dtype=torch.uint8, device="cuda")
            sc = torch.full((rows * 4 + 64,), 0xAA, dtype=torch.uint8, device="cuda")
            quantize_qk(xb, out, sc, mul=mul)
            torch.cuda.synchronize()
            want, want_sc = oracle.quantize_rows(xf, np.float32(mul))
            assert np.array_equal(sc.cpu().numpy()[: rows * 4].reshape(rows, 4), want_sc), (rows, mul)
            assert np.array_equal(out.cpu().numpy(), want), (rows, mul)
            assert (sc.cpu().numpy()[rows * 4:] == 0xAA).all()      # nothing written past the rows
    for n in (8, 128 * 77, 128 * 4096 + 8):
        x = (rng.standard_normal(n) * 3.0).astype(np.float32)
        xb = torch.from_numpy(x).to(torch.bfloat16).cuda()
        out = torch.empty(n, dtype=torch.uint8, device="cuda")
        vd = torch.zeros(1024, dtype=torch.float32, device="cuda")
        quantize_v(xb, out, vd)
        torch.cuda.synchronize()
        want, want_vd = oracle.quantize_tensor(xb.float().cpu().numpy())
        assert float(vd[0]) == np.float32(want_vd) and np.array_equal(out.cpu().numpy(), want), n
    z = torch.zeros(64, dtype=torch.bfloat16, device="cuda")
    out = torch.full((64,), 0xAA, dtype=torch.uint8, device="cuda")
    vd = torch.zeros(2, dtype=torch.float32, device="cuda")
    quantize_v(z, out, vd)
    assert float(vd[0]) == 1.0 and not out.cpu().numpy().any()


@pytest.mark.gpu
def test_quantise_then_attend_passes_the_gate(oracle):
    """bf16 Q, K, V -> device quantisers -> attention, scored like every other shape: against the fp64 oracle on the quantised operands
    and the reference path's error on the same operands."""
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import Q_PRESCALE, fmha_fwd_mxfp8, quantize_qk, quantize_v
    B, H, HK, S, SK = 1, 4, 2, 300, 1337
    g = torch.Generator().manual_seed(11)
    q = torch.randn(B, S, H, 128, generator=g).to(torch.bfloat16).cuda()
    k = torch.randn(B, SK, HK, 128, generator=g).to(torch.bfloat16).cuda()
    v = torch.randn(B, SK, HK, 128, generator=g).to(torch.bfloat16).cuda()
    q8, k8, v8 = (torch.empty(t.shape, dtype=torch.uint8, device="cuda") for t in (q, k, v))
    qs = torch.zeros(B * S * H * 4 + 512 * H * 4, dtype=torch.uint8, device="cuda")
    ks = torch.zeros(B * SK * HK * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda")
    vs = torch.zeros(1024, dtype=torch.float32, device="cuda")
    quantize_qk(q, q8, qs, mul=Q_PRESCALE)
    quantize_qk(k, k8, ks)
    quantize_v(v, v8, vs)
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    fmha_fwd_mxfp8(q8, k8, v8, qs, ks, vs, out)
    torch.cuda.synchronize()
    inp = oracle.Inputs(B, H, HK, S, SK, q8.cpu().numpy(), k8.cpu().numpy(), v8.cpu().numpy(), qs.cpu().numpy(), ks.cpu().numpy(), float(vs[0]))
    rows = 32
    ref = oracle.reference(inp, rows)
    ours = oracle.compare(inp, out.view(torch.int16).cpu().numpy().view(np.uint16), ref, rows)
    theirs = oracle.compare(inp, oracle.recipe_forward(inp, rows, 0), ref, rows)
    assert ours.bad <= theirs.bad and ours.mean_err <= 1.10 * theirs.mean_err and ours.worst_err <= 2e-2, (ours, theirs)
    # and the quantised attention is close to plain bf16 attention on the unquantised tensors (a sanity bound, not a gate)
    qf, kf, vf = q.float(), k.float().repeat_interleave(H // HK, dim=2), v.float().repeat_interleave(H // HK, dim=2)
    s = torch.einsum("bshd,bthd->bhst", qf, kf) / 128 ** 0.5
    want = torch.einsum("bhst,bthd->bshd", torch.softmax(s, -1), vf)
    assert (out.float() - want).abs().max().item() < 0.05


def test_the_division_by_a_residual_rounds_like_a_division():
    """The device quantiser of V divides by amax / 448 with a reciprocal and one residual correction. x and amax are bf16, so their 128 x 128
    mantissas are all there is, with either sign, and the two zeros: the corrected quotient is the correctly rounded one for each, bit for bit."""
    f32, f64 = np.float32, np.float64
    x = (128 + np.arange(128)).astype(f32)
    x = np.concatenate([x, -x, np.array([0.0, -0.0], f32)])[None, :]
    vd = ((128 + np.arange(128)).astype(f32) / f32(448))[:, None]
    r = f32(1) / vd
    q = x * r
    rem = (q.astype(f64) * vd.astype(f64) - x.astype(f64)).astype(f32)   # the products of two f32 and the difference are exact in f64
    fixed = (-rem.astype(f64) * r.astype(f64) + q.astype(f64)).astype(f32)
    assert (q != x / vd).any() and np.array_equal(fixed.view(np.uint32), (x / vd).view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("n_vec", [16, 32769, 1212416])   # one launch; the general form with one and with four loads per thread
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -110])   # the divisor inside the range of the correction, and below it
def test_quantize_v_keeps_the_sign_of_zero(n_vec, scale):
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import quantize_v
    x = torch.tensor([0.0, -0.0, 1.0, -1.0, 2.0 ** -20, -(2.0 ** -20), -0.0, 0.0]).repeat(n_vec).mul(scale).to(torch.bfloat16)
    out, vs = torch.zeros(n_vec * 8, dtype=torch.uint8, device="cuda"), torch.zeros(2, dtype=torch.float32, device="cuda")
    quantize_v(x.cuda(), out, vs)
    # +-448 are the bytes 0x7E and 0xFE; 2^-20 of them are below half the smallest e4m3 step
    assert torch.equal(out.cpu(), torch.tensor([0x00, 0x80, 0x7E, 0xFE, 0x00, 0x80, 0x80, 0x00], dtype=torch.uint8).repeat(n_vec))


@pytest.mark.gpu
@pytest.mark.parametrize("n_vec", [1, 31, 8191, 8193, 32768, 32769, 1212416, 1212417])   # a cluster's registers full and one more; one and four loads per thread
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -110])   # the divisor inside the range of the correction, and below it
def test_quantize_v_sizes(oracle, n_vec, scale):
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import quantize_qk, quantize_v
    x = (torch.randn(n_vec * 8, generator=torch.Generator().manual_seed(n_vec)) * scale).to(torch.bfloat16)
    out, vs = torch.zeros(n_vec * 8, dtype=torch.uint8, device="cuda"), torch.zeros(1024, dtype=torch.float32, device="cuda")
    quantize_v(x.cuda(), out, vs)
    vd = (x.float().abs().max() / 448.0).item()
    assert vs[0].item() == vd
    want = (x.float() / vd).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    assert torch.equal(out.cpu(), want)
    if n_vec % 16 == 0 and scale == 1.0:   # whole rows of 128: the Q / K quantiser at the same sizes
        rows = n_vec // 16
        y, s = torch.zeros(rows, 128, dtype=torch.uint8, device="cuda"), torch.zeros(rows * 4, dtype=torch.uint8, device="cuda")
        quantize_qk(x.view(rows, 128).cuda(), y, s, mul=1.0)
        f = x.view(rows, 4, 32).float()
        e = (torch.frexp(f.abs().amax(-1)).exponent - 1 - 8 + 127).clamp(0, 254)
        assert torch.equal(s.cpu().view(rows, 4).int(), e.int())
        assert torch.equal(y.cpu(), torch.ldexp(f, (127 - e)[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8).view(rows, 128))


@pytest.mark.gpu
def test_small_v_back_to_back(oracle):
    """The one-launch form, each launch allowed to start while the one before it runs: 64 tensors of different magnitudes and sizes on one stream without a
    wait in between. A maximum that one CTA of a cluster misses (its neighbours write it into its shared memory) shows in its bytes and the descale."""
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import quantize_v
    g = torch.Generator().manual_seed(9)
    sizes = [8 * n for n in (1, 1000, 8192, 8193, 20000, 32768)]
    xs = [(torch.randn(sizes[i % 6], generator=g) * 2.0 ** (i % 11 - 5)).to(torch.bfloat16) for i in range(64)]
    for x in xs:   # the maximum in another CTA's share each time
        x[torch.randint(0, x.numel(), (1,), generator=g)] = 7.0 * x.float().abs().max().item()
    dev = [x.cuda() for x in xs]
    outs = [torch.zeros(x.numel(), dtype=torch.uint8, device="cuda") for x in xs]
    vs = [torch.zeros(2, dtype=torch.float32, device="cuda") for _ in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for x, out, v in zip(dev, outs, vs):
            quantize_v(x, out, v)
    torch.cuda.synchronize()
    for x, out, v in zip(xs, outs, vs):
        vd = (x.float().abs().max() / 448.0).item()
        assert v[0].item() == vd
        assert torch.equal(out.cpu(), (x.float() / vd).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 8, 2, 1000, 1000), (1, 2, 2, 200, 300), (2, 8, 2, 1, 4096), (1, 4, 4, 300, 2100), (1, 8, 8, 512, 4500)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("captured", [False, True])
def test_a_chain_of_dependent_launches_reads_what_the_one_before_wrote(shape, captured):
    """quantise -> attend, eight times over the same operand buffers with data of another magnitude each time and no wait in between (the kernels of the chain
    may start while the one before them runs, so a scale read too early would be the last step's), against the same calls with a wait behind each."""
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import Q_PRESCALE, device_status, fmha_fwd_mxfp8, quantize_qk, quantize_v
    B, H, HK, S, SK = shape
    g = torch.Generator(device="cuda").manual_seed(21)
    data = [[(torch.randn(dims, generator=g, device="cuda") * 2.0 ** e).to(torch.bfloat16) for dims, e in (((B, S, H, 128), i % 3 - 2), ((B, SK, HK, 128), -(i % 2)), ((B, SK, HK, 128), 4 - i))]
            for i in range(8)]
    q8, k8, v8 = (torch.empty(x.shape, dtype=torch.uint8, device="cuda") for x in data[0])
    qs = torch.zeros(B * S * H * 4 + 512 * H * 4, dtype=torch.uint8, device="cuda")
    ks = torch.zeros(B * SK * HK * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda")
    vs = torch.zeros(1024, dtype=torch.float32, device="cuda")

    def chain(outs, wait):
        for (q, k, v), out in zip(data, outs):
            for call in (lambda: quantize_qk(q, q8, qs, mul=Q_PRESCALE), lambda: quantize_v(v, v8, vs), lambda: quantize_qk(k, k8, ks),
                         lambda: fmha_fwd_mxfp8(q8, k8, v8, qs, ks, vs, out)):
                call()
                wait()

    want, got = ([torch.zeros(B, S, H, 128, dtype=torch.bfloat16, device="cuda") for _ in data] for _ in range(2))
    chain(want, torch.cuda.synchronize)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(got, lambda: None)   # (first calls: workspaces and tensor maps)
        torch.cuda.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                chain(got, lambda: None)
        for _ in range(10):
            for x in got:
                x.zero_()
            graph.replay() if captured else chain(got, lambda: None)
            torch.cuda.synchronize()
            assert all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(got, want))
    assert device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [75775, 75776, 94719, 94720, 94721, 189441, 284161])   # the wide form from its first size on; one round of its grid's loop on 148 SMs, a row more, two and three
def test_quantize_qk_rounds_of_the_wide_form(rows):
    torch = pytest.importorskip("torch")
    from amdgpu_rustdsl_b200 import quantize_qk
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(rows, 128, generator=g, device="cuda") * torch.exp2(torch.randint(-12, 12, (rows, 1), generator=g, device="cuda").float())).to(torch.bfloat16)
    y, s = torch.full((rows + 1, 128), 0xAA, dtype=torch.uint8, device="cuda"), torch.full((rows * 4 + 16,), 0xAA, dtype=torch.uint8, device="cuda")
    quantize_qk(x, y[:rows], s)
    f = x.view(rows, 4, 32).float()
    e = (torch.frexp(f.abs().amax(-1)).exponent - 1 - 8 + 127).clamp(0, 254)
    assert torch.equal(s[: rows * 4].view(rows, 4).int(), e.int())
    want = torch.ldexp(f, (127 - e)[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8).view(rows, 128)
    assert torch.equal(y[:rows], want)
    assert (y[rows] == 0xAA).all() and (s[rows * 4:] == 0xAA).all()   # nothing written past the rows
