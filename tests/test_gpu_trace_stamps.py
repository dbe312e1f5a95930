"""The time stamps of an attached trace buffer: the copies and the matrix instructions of every key tile leave theirs, the first tile's too."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STAMP_WORD = 16384 + 16384 + 256 + 4096   # first word of the stamps: [role 4][tile 32][slot 8] 64-bit clock values
ROLE_QK, ROLE_PV = 2, 3
SLOT_MMA, SLOT_ISSUED, SLOT_COPY = 2, 4, 6


@pytest.mark.parametrize("SK,path,splits", [(384, "t128", None), (1100, "vs128", None), (2048, "kvsplit", 2)])   # both softmax recipes, the split kernel
def test_every_tile_leaves_its_stamps(abi, SK, path, splits):
    from amdgpu_rustdsl_b200 import device_status, fmha_fwd_mxfp8
    lib, S = abi.load(), 128
    q, k, v = (torch.full((1, n, 1, 128), 0x38, dtype=torch.uint8, device="cuda") for n in (S, SK, SK))
    qs, ks = (torch.full((4 * n + 640 * 4,), 127, dtype=torch.uint8, device="cuda") for n in (S, SK))
    vs = torch.ones(1024, dtype=torch.float32, device="cuda")
    out = torch.empty((1, S, 1, 128), dtype=torch.bfloat16, device="cuda")
    buf = torch.full((abi.TRACE_BYTES // 4,), -1, dtype=torch.int32, device="cuda")
    assert lib.fmha_mxfp8_trace_attach(buf.data_ptr(), abi.TRACE_BYTES) == 0
    try:
        fmha_fwd_mxfp8(q, k, v, qs, ks, vs, out, path=path, splits=splits)
        torch.cuda.synchronize()
    finally:
        lib.fmha_mxfp8_trace_attach(None, 0)
    stamps = buf[STAMP_WORD:].view(torch.int64).view(4, 32, 8).cpu()
    tiles = -(-SK // 128) // (splits or 1)   # of the first item
    for role in (ROLE_QK, ROLE_PV):
        for tile in range(tiles):
            copy, mma, issued = (int(stamps[role, tile, slot]) for slot in (SLOT_COPY, SLOT_MMA, SLOT_ISSUED))
            assert -1 not in (copy, mma, issued), (role, tile, "no stamp")
            assert copy <= mma <= issued, (role, tile)   # one SM's clock: the tile's copy is sent out before it is multiplied
    assert (stamps[ROLE_QK, tiles:24, SLOT_COPY] == -1).all()
    assert device_status() == 0
