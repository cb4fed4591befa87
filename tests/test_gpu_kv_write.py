"""Keys and values into their pages: by 16-byte pieces where rows allow, else by elements."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# pieces of a token against the threads of a block: one; fewer than a warp; both held pieces and some behind them; heads of odd pieces; no pieces
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("nk,dk,nv,dv", [(1, 8, 1, 8), (2, 24, 1, 40), (8, 64, 4, 128), (16, 128, 8, 256), (3, 72, 2, 192), (2, 20, 3, 12), (1, 7, 1, 9)])
@pytest.mark.parametrize("shift", [0, 1])
def test_keys_and_values_into_pages(dtype, nk, dk, nv, dv, shift):
    from prelude_b200.ops import kernels as K
    T, page, pages = 37, 16, 9
    proj = torch.randn(T, shift + nk * dk + nv * dv + 8, device=DEV).to(dtype)
    k, v = proj[:, shift:shift + nk * dk], proj[:, shift + nk * dk:shift + nk * dk + nv * dv]
    table = torch.tensor([[7, 1, 4], [2, 8, 3]], dtype=torch.int32, device=DEV)
    row = torch.tensor([0] * 20 + [1] * 15 + [-1] * 2, dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(20) + 11, torch.arange(15) + 29, torch.zeros(2)]).int().to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kp, vp = torch.full((pages, nk, page, dk), 5.0, dtype=dtype, device=DEV), torch.full((pages, nv, page, dv), 6.0, dtype=dtype, device=DEV)
    want = [kp.cpu(), vp.cpu()]
    for n in range(35):
        p, at = int(table[int(row[n]), int(pos[n]) // page]), int(pos[n]) % page
        for pages_, x, h, d in ((want[0], k, nk, dk), (want[1], v, nv, dv)):
            e = torch.arange(d)
            to = ((e // 8) ^ (at & 7)) * 8 + e % 8 if K.kv_swizzled(dtype, d) else e
            pages_[p, :, at, to] = x[n].view(h, d).cpu()
    K.kv_write_pages(k, v, kp, vp, pos, row, table, status)
    assert torch.equal(kp.cpu(), want[0]) and torch.equal(vp.cpu(), want[1]) and int(status) == 0
    before = kp.clone(), vp.clone()
    K.kv_write_pages(k[:1], v[:1], kp, vp, pos, row, torch.full_like(table, pages), status)       # a page that is not there
    assert int(status) == 2 and torch.equal(kp, before[0]) and torch.equal(vp, before[1])
