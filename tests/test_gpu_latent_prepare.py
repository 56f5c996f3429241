"""GPU: the pass that makes latent cache rows and turned queries ready, in 4-value pieces, against the general kernel, which
inputs off the pieces take: ranks below the CTA's width, a turned part below the rotary width, few rows.  Both compute in
fp32 in another order of at most 512 squares (2^-18 of the value) and round once: one ulp of the type."""
import pytest
import torch

from scalellm_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
ULP = {torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10, torch.float32: 2.0 ** -18}


def _close(a, b, ulp):
    assert bool(torch.isfinite(a).all())
    a, b = a.double(), b.double()
    assert bool(((a - b).abs() <= ulp * b.abs() + 2.0 ** -18).all()), float((a - b).abs().max())


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", list(ULP))
@pytest.mark.parametrize("rows,H,dim,rd,dims,rank", [(1, 1, 128, 64, 64, 512), (9, 16, 128, 64, 64, 512), (5, 3, 64, 32, 24, 100),
                                                     (3, 2, 0, 8, 4, 4)])
def test_latent_inputs(rows, H, dim, rd, dims, rank, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    nq, nd = H * (dim + rd), rank + rd
    q0, d0 = rnd(rows, nq).to(dtype), rnd(rows, nd).to(dtype)
    w, freq = 1.0 + 0.2 * rnd(rank), torch.rand(dims // 2, generator=g, device=DEV)
    pos, slots = _i32([5 * i for i in range(rows)]), _i32(list(range(rows, 0, -1)))
    got = []
    for shift in (0, 1):
        q = torch.zeros(rows, nq + 4, dtype=dtype, device=DEV)[:, shift: shift + nq]
        d = torch.zeros(rows, (nd + 3) // 4 * 4 + 4, dtype=dtype, device=DEV)[:, shift: shift + nd]
        q.copy_(q0)
        d.copy_(d0)
        cache = torch.full((rows + 2, nd), 9.0, dtype=dtype, device=DEV)
        kernels.latent_prepare(q, d, cache, w, freq, 1.5, pos, slots, H, dim, rd, dims, rank, 1e-6)
        got.append((q, cache))
    _close(got[0][0], got[1][0], ULP[dtype])
    _close(got[0][1], got[1][1], ULP[dtype])
