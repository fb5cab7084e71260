"""The per-update kernels' order of a plane's cells: those outside the z faces first in double precision
and, for Bloch pairs, where the z extent and its faces are multiples of 8, else row by row. A grid with y and z exchanged
has the same physics mirrored, and its y faces do not touch the order: fields of both after a few steps,
with faces at either end, both, of unequal or nearly full depth."""
import copy

import numpy
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# z extent, n and p thickness: split for Bloch pairs, in double only, not at all; nearly all cells in faces
Z = [(24, 8, 8), (40, 8, 0), (40, 0, 16), (64, 24, 32), (16, 8, 0), (25, 8, 8), (24, 4, 8), (9, 8, 0), (9, 0, 1), (7, 3, 4), (5, 0, 0),
     (300, 8, 16)]


@pytest.mark.parametrize("dtype", [numpy.float32, numpy.float64])
@pytest.mark.parametrize("sz,tn,tp", Z)
@pytest.mark.parametrize("form", ["plain", "mu", "bloch"])
def test_z_order(sz, tn, tp, dtype, form):
    from opencl_fdtd_gb300 import Simulation
    rng = numpy.random.default_rng(sz + tn)
    shape = (5, 6, sz)
    eps = [rng.uniform(1, 4, shape).astype(dtype) for _ in range(3)]
    init = {k: [rng.standard_normal(shape).astype(dtype) for _ in range(3)] for k in "EH"}
    mu = [rng.uniform(1, 2, shape).astype(dtype) for _ in range(3)] if form != "plain" else None
    pmls = [{"axis": "z", "polarity": p, "thickness": t} for p, t in (("n", tn), ("p", tp)) if t]
    pmls += [{"axis": "x", "polarity": "n", "thickness": 2}]
    if form != "bloch":
        pmls += [{"axis": "y", "polarity": "p", "thickness": 3}]

    def swap(fields):
        # exchanging two axes mirrors space: E -> (Ex, Ez, Ey), H -> -(Hx, Hz, Hy)
        return [numpy.ascontiguousarray(fields[c].swapaxes(1, 2)) for c in (0, 2, 1)]

    def build(sw):
        ax = {"x": "x", "y": "z", "z": "y"}
        kw = dict(epsilon=swap(eps) if sw else eps, float_type=dtype, do_poynting=False,
                  pmls=[dict(p, axis=ax[p["axis"]]) if sw else dict(p) for p in pmls],
                  initial_fields={"E": swap(init["E"]) if sw else init["E"],
                                  "H": [-f for f in swap(init["H"])] if sw else init["H"]})
        if mu is not None:
            kw["mu"] = swap(mu) if sw else mu
        if form == "bloch":
            kw["bloch_boundaries"] = [{"axis": "z" if sw else "y", "real": 0.8, "imag": 0.6}]
        return Simulation(**copy.deepcopy(kw))
    a, b = build(False), build(True)
    a.run(4, path="plain")
    b.run(4, path="plain")

    def parts(sim, name, sw):
        f = [v.cpu().numpy().astype(float) for v in getattr(sim, name).view(3, *(shape if not sw else (5, sz, 6)))]
        return [f[c].swapaxes(1, 2) for c in (0, 2, 1)] if sw else f
    # four steps of at most about 30 roundings each on values of order 10
    tol = 4 * 30 * numpy.finfo(dtype).eps * 16
    for name in ("E", "H") + (("F", "G") if form == "bloch" else ()):
        sign = -1.0 if name in "HG" else 1.0
        for u, v in zip(parts(a, name, False), parts(b, name, True)):
            assert abs(u - sign * v).max() <= tol, name
