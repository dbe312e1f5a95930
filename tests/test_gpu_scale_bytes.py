"""The scale byte of every query row and key reaches the product it belongs to: rows whose scale lets one key with a larger scale carry the whole row, beside
rows whose scale makes all keys alike."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,SK,H,HK", [(1, 33, 1, 1), (5, 131, 4, 1), (130, 257, 2, 2), (3, 700, 8, 2), (129, 641, 3, 3), (257, 1025, 4, 2)])
@pytest.mark.parametrize("v_blocks", [False, True])
def test_every_scale_byte(S, SK, H, HK, v_blocks):
    from amdgpu_rustdsl_b200 import device_status, fmha_fwd_mxfp8
    edges = sorted({t for t in (0, 31, 32, 63, 64, 95, 96, 127, 128, 159, 255, 256, 511, 512, 639, 640, SK - 1) if t < SK})   # of lanes' words and of tiles
    B, g = len(edges), H // HK
    gen = torch.Generator(device="cuda").manual_seed(S * SK + H)
    one = 0x38   # e4m3 1.0: a score is 128 x 2^(scale of the row + scale of the key)
    q, k = torch.full((B, S, H, 128), one, dtype=torch.uint8, device="cuda"), torch.full((B, SK, HK, 128), one, dtype=torch.uint8, device="cuda")
    v = torch.randn((B, SK, HK, 128), generator=gen, device="cuda").to(torch.float8_e4m3fn)
    key = (torch.tensor(edges, device="cuda")[:, None] + 7 * torch.arange(HK, device="cuda")) % SK   # [B, HK]: the key that carries the rows
    ks = torch.zeros(B * SK * HK * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda")
    ks4 = ks[: B * SK * HK * 4].view(B, SK, HK, 4)
    ks4.fill_(127 - 4)                                                     # scores of 8 ...
    ks4.scatter_(1, key[:, None, :, None].expand(B, 1, HK, 4), 127 - 1)    # ... and one of 64: the others weigh 2^-56
    qs = torch.zeros(B * S * H * 4 + 512 * H * 4, dtype=torch.uint8, device="cuda")
    qs4 = qs[: B * S * H * 4].view(B, S, H, 4)
    flat = (torch.arange(S, device="cuda")[:, None] + torch.arange(H, device="cuda")) % 3 == 1   # [S, H]: rows with scores of next to nothing
    qs4.copy_(torch.where(flat, 127 - 20, 127).to(torch.uint8)[None, :, :, None].expand(B, S, H, 4))
    vs = torch.ones(1024, dtype=torch.float32, device="cuda")
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    vb = torch.full((B, -(-SK // 32), HK, 128), 127, dtype=torch.uint8, device="cuda") if v_blocks else None
    fmha_fwd_mxfp8(q, k, v.view(torch.uint8), qs, ks, vs, out, v_blockscale=vb)
    vf = v.double()
    carried = vf.gather(1, key[:, None, :, None].expand(B, 1, HK, 128)).repeat_interleave(g, 2)   # [B, 1, H, 128]
    want = torch.where(flat[None, :, :, None], vf.mean(1, keepdim=True).repeat_interleave(g, 2), carried)
    # All weights of a flat row are the same power of two, and so is the one of a carried row: what is left is the f32 sum of up to 1025 products (2^-24 x
    # sqrt(1025) x max|v| < 1e-5) and the rounding to bf16
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
    assert device_status() == 0


# (B, S, SK, H, HK, path, splits, causal): short and long recipe, packed heads; launches of which a CTA walks four items (the Q scales' two buffers come
# round again from its third on); few items, cut between the CTAs of clusters; a last round cut in two; splits, whose items start at other keys; the mask, whose
# items come in an order of their own
WORDS = [(4, 33, 300, 2, 2, "t128", None, False), (4, 257, 513, 48, 48, "vs128", None, False), (16, 130, 641, 48, 12, "vs128", None, False),
         (4, 5, 2500, 4, 1, "t128", None, False), (4, 200, 6200, 20, 20, "vs128", None, False), (4, 200, 1700, 4, 2, "kvsplit", 4, False),
         (4, 130, 1998, 3, 3, "kvsplit", 8, False), (4, 300, 700, 4, 2, "vs128", None, True), (4, 641, 641, 40, 20, "vs128", None, True)]


@pytest.mark.parametrize("B,S,SK,H,HK,path,splits,causal", WORDS)
@pytest.mark.parametrize("v_blocks", [False, True])
def test_every_byte_of_a_scale_word(B, S, SK, H, HK, path, splits, causal, v_blocks):
    """Batch element b has data in the 32 columns of byte b % 4 only. There a key's byte says whether it carries the rows (score 64) or weighs nothing (8), and a row's
    whether it sees that or all keys alike, each drawn for every row, key and byte: a byte of another place in the word, row, key or head gives another mean."""
    from amdgpu_rustdsl_b200 import device_status, fmha_fwd_mxfp8
    if v_blocks and causal:
        pytest.skip("the mask has no form with V block scales")
    gen, g = torch.Generator(device="cuda").manual_seed(B * S * SK + H), H // HK
    q, k = torch.zeros((B, S, H, 128), dtype=torch.uint8, device="cuda"), torch.zeros((B, SK, HK, 128), dtype=torch.uint8, device="cuda")
    for b in range(B):
        for x in (q, k):
            x[b, :, :, 32 * (b % 4): 32 * (b % 4) + 32] = 0x38   # e4m3 1.0: a score is 32 x 2^(byte of the row + byte of the key)
    v = torch.randn((B, SK, HK, 128), generator=gen, device="cuda").to(torch.float8_e4m3fn)
    carries = torch.rand((B, SK, HK, 4), generator=gen, device="cuda") < 0.5
    alike = torch.rand((B, S, H, 4), generator=gen, device="cuda") < 0.5
    qs, ks = (torch.zeros(n * 4 + 640 * H * 4, dtype=torch.uint8, device="cuda") for n in (B * S * H, B * SK * HK))
    ks[: carries.numel()] = torch.where(carries, 127 + 1, 127 - 2).to(torch.uint8).flatten()
    qs[: alike.numel()] = torch.where(alike, 127 - 60, 127).to(torch.uint8).flatten()
    vs = torch.ones(1024, dtype=torch.float32, device="cuda")
    out = torch.full((B, S, H, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    vb = torch.full((B, -(-SK // 32), HK, 128), 127, dtype=torch.uint8, device="cuda") if v_blocks else None
    assert fmha_fwd_mxfp8(q, k, v.view(torch.uint8), qs, ks, vs, out, path=path, splits=splits, causal=causal, v_blockscale=vb) == (path, splits or 0)

    byte = torch.arange(B, device="cuda") % 4
    w = torch.stack([carries[b, :, :, byte[b]] for b in range(B)]).double()[..., None]   # [B, SK, HK, 1]
    flat = torch.stack([alike[b, :, :, byte[b]] for b in range(B)])[..., None]           # [B, S, H, 1]
    vf = v.double()
    last = torch.arange(S, device="cuda") + (SK - S) if causal else torch.full((S,), SK - 1, device="cuda")   # a row's last key

    def upto(x):   # sums over a row's keys
        return (x.cumsum(1)[:, last] if causal else x.sum(1, keepdim=True).expand(-1, S, -1, -1)).repeat_interleave(g, 2)

    seen = (last + 1).double()[None, :, None, None]
    n, total = upto(w), upto(vf) / seen
    want = torch.where(flat | (n == 0), total, upto(w * vf) / n.clamp(min=1))   # (a row none of whose keys carries: all weigh alike)
    # The weights of a row are one power of two, or 2^-56 of it, and the f32 sums of up to 6200 products of e4m3 numbers with them are exact: the rounding to bf16 is
    # left, and for splits the one of their means to f16 (2^-11 of the largest) and what two log-sum-exps of about 75 in f32 lose (2^-16 of it)
    bound = want.abs() * 2.0 ** -8 + 1e-5
    if splits:
        run = -(-(-(-SK // 128)) // splits) * 128
        for lo in range(0, SK, run):
            vp, wp = vf[:, lo:lo + run], w[:, lo:lo + run]
            for mean in (vp.mean(1, keepdim=True), (vp * wp).sum(1, keepdim=True) / wp.sum(1, keepdim=True).clamp(min=1)):
                bound = torch.maximum(bound, want.abs() * 2.0 ** -8 + 1e-5 + mean.abs().repeat_interleave(g, 2) * (2.0 ** -11 + 2.0 ** -16))
    wrong = ~((out.double() - want).abs() <= bound)
    assert not wrong.any(), (int(wrong.sum()), wrong.nonzero()[:4].tolist())
    assert device_status() == 0
