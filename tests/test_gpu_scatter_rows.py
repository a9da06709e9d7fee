"""The per-plane scatter that takes its plan as kernel parameters (at most 8 stores, rows of at most 8 outputs, no expressions) and the one
that reads it from memory, at the edges of both rules, bit for bit against the CPU interpreter."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import fortis_b200
from fortis_b200 import descriptors as D
from oracle import fortis_oracle as fo


@pytest.mark.parametrize("elt", ["f32", "f64"])
@pytest.mark.parametrize("nx,ny,nout,nstores", [(1, 1, 1, 1), (127, 1, 3, 3), (32, 4, 3, 8), (43, 3, 8, 8), (43, 3, 8, 9), (43, 3, 9, 8), (150, 130, 2, 3)])
def test_planes(nx, ny, nout, nstores, elt):
    nz = 3
    G, S, Lp, K = D.stencil(nx, ny, nz, nfields=1, nout=nout)
    S["arrays"] = [dict(S["arrays"][0], name="o%d" % q, ssa="%%o%d" % q, elt=elt) for q in range(nstores)]
    S["stores"] = [{"slot": (3 * q) % nout, "array": q, "idx": [["i", q % 3 - 1], ["j", 0], ["v", 0]]} for q in range(nstores)]
    layers = fortis_b200.mlp_layers([9, 16, nout], seed=2, act="relu", bias="uniform")
    h = fortis_b200.Host()
    h.reset()
    h.configure(gather=G, scatter=S, loop=Lp, kdist=K)
    h.load_model(fortis_b200.write_blob(layers))
    x = torch.randn((nz, ny + 2, nx + 2), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))
    out = [torch.full((nz, ny + 2, nx + 2), 7.0, device="cuda", dtype=torch.float32 if elt == "f32" else torch.float64) for _ in range(nstores)]
    h.gather([x])
    h.forward_batched()
    Y = h.model_output(nx * ny * nz, nout)
    ref = [np.full((nx + 2, ny + 2, nz), 7.0, np.float32 if elt == "f32" else np.float64, order="F") for _ in range(nstores)]
    for k in (2, 1, 3):
        h.scatter(out, args=(k,))
        fo.scatter(S, Lp, K, Y, ref, args=(k,))
    h.sync()
    for a, b in zip(out, ref):
        assert np.array_equal(a.cpu().numpy().reshape(-1), b.reshape(-1, order="F"))
    h.reset()
