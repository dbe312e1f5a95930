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
