"""The fused stencil step at the edges of its tiles (32 x 4 points), of its grid (more tiles than resident blocks, whose coordinates are
advanced with carries) and with outputs stored in another order, against float64.

Tolerance: sums of at most 27 fp32 products per layer, three layers: below 3 * 27 * 2^-24 = 4.9e-6 of the largest terms; 5e-6 of the
result's 2-norm is what the other stencil tests ask for."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors as D


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 0, 1), (1,)])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (32, 4, 1), (33, 5, 3), (31, 3, 2), (70, 1, 5), (1, 90, 2), (645, 515, 3)])
def test_stencil_tiles(nx, ny, nz, order):
    h = fortis_b200.Host()
    h.reset()
    layers = fortis_b200.mlp_layers([27, 20, 20, 3], seed=4, init="uniform", act="relu", bias="uniform")
    G, S, Lp, K = D.stencil(nx, ny, nz)
    S["arrays"] = S["arrays"][:len(order)]
    S["stores"] = [dict(S["stores"][q], slot=s) for q, s in enumerate(order)]
    h.configure(gather=G, scatter=S, loop=Lp, kdist=K)
    h.option("checksum", 1)
    h.load_model(fortis_b200.write_blob(layers))
    g = torch.Generator(device="cuda").manual_seed(nx * 7 + ny)
    f = [torch.randn((nz, ny + 2, nx + 2), device="cuda", generator=g) for _ in range(3)]
    out = [torch.full_like(f[0], 7.0) for _ in order]
    h.step(f, out)
    h.sync()
    x = torch.stack([a[:, 1 + dj:1 + dj + ny, 1 + di:1 + di + nx] for a in f for dj in (-1, 0, 1) for di in (-1, 0, 1)], dim=-1).double()
    for l in layers:
        x = x @ torch.from_numpy(l["W"]).cuda().double().T + torch.from_numpy(l["b"]).cuda().double()
        if l["act"] == "relu":
            x = x.clamp_min(0)
    total = 0.0
    for a, s in zip(out, order):
        got = a[:, 1:-1, 1:-1].double()
        assert float((got - x[..., s]).norm()) <= 5e-6 * float(x[..., s].norm())
        total += float(got.sum())
        a[:, 1:-1, 1:-1] = 7.0
        assert bool((a == 7.0).all())                            # the halo is not written
    assert abs(h.step_checksum() - total) <= 1e-9 * max(1.0, abs(total)) * nx * ny * nz
    h.reset()
