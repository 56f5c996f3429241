"""Router and combine of the token-choice experts (csrc/moe.cu) at the sizes where their loads change shape: rows that are
and are not 16-byte pieces, fewer and more experts than warps and lanes, ties, infinities, all experts chosen."""
import pytest
import torch

from scalellm_b200 import kernels

pytestmark = pytest.mark.gpu
DT = {torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -22}


@pytest.mark.parametrize("rows,W,E,top", [(1, 64, 4, 2), (3, 2048, 8, 2), (16, 132, 33, 5), (2, 130, 9, 9), (5, 61, 70, 3)])
@pytest.mark.parametrize("dtype", list(DT))
def test_route(rows, W, E, top, dtype):
    g = torch.Generator(device="cuda").manual_seed(W + E)
    h = torch.randn(rows, W + 4, generator=g, device="cuda").to(dtype)[:, :W]
    R = torch.randn(E, W, generator=g, device="cuda")
    R[E - 1] = R[0]                                             # a tie: the first index wins
    ids, wts = kernels.moe_route(h, R, top)
    z = h.double() @ R.double().T
    want = torch.sort(z, dim=1, descending=True, stable=True)
    for r in range(rows):
        got = ids[r].long()
        # fp32 sums of W products: an order may differ only where logits are that close
        slack = W * 2.0 ** -24 * float((h[r].double().abs() @ R.double().abs().T).max())
        assert len(set(got.tolist())) == top
        assert bool(((z[r, got] - want.values[r, :top]).abs() <= 2 * slack).all())
        if 0 in got.tolist() and E - 1 in got.tolist():
            assert got.tolist().index(0) < got.tolist().index(E - 1)
        assert E - 1 not in got.tolist() or 0 in got.tolist()
        ref = torch.sigmoid(z[r, got])
        assert bool(((wts[r].double() - ref).abs() <= slack + 2.0 ** -21).all())


def test_route_of_infinite_logits():
    h = torch.ones(1, 8, dtype=torch.float32, device="cuda")
    R = torch.zeros(3, 8, device="cuda")
    R[0], R[1], R[2] = -float("inf"), 1.0, float("nan")
    ids, wts = kernels.moe_route(h, R, 2)
    assert ids.tolist() == [[1, 0]] and float(wts[0, 1]) == 0.0


@pytest.mark.parametrize("rows,W,top,addend", [(1, 8, 1, False), (3, 2056, 2, True), (2, 2050, 3, True), (1030, 40, 2, False),
                                                (2, 100000, 5, True)])
@pytest.mark.parametrize("dtype", list(DT))
def test_combine(rows, W, top, addend, dtype):
    g = torch.Generator(device="cuda").manual_seed(W)
    y = torch.randn(rows * top, W, generator=g, device="cuda").to(dtype)
    pos = torch.randperm(rows * top, generator=g, device="cuda").to(torch.int32)
    add = torch.randn(rows, W, generator=g, device="cuda").to(dtype) if addend else None
    out = kernels.moe_combine(y, pos, rows, top, 0.5, add)
    terms = y.double()[pos.long()].view(rows, top, W)
    ref, mag = 0.5 * terms.sum(1), 0.5 * terms.abs().sum(1)
    if addend:
        ref, mag = ref + add.double(), mag + add.double().abs()
    assert bool(((out.double() - ref).abs() <= DT[dtype] * ref.abs() + (top + 2) * 2.0 ** -24 * mag + 1e-30).all())
