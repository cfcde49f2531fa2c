"""The step kernels on boxes of quads, bit for bit against the oracle where they can go
wrong: rows that end inside a quad, faces of the CPML frame that share one or leave less
than two between them, boxes that reach past the grid in every axis, both ways of reading
neighbours; velocity rings of every length; dividends from subnormal to overflowing and
divisors outside the fast division's range."""
import numpy as np
import pytest

from ifosb import synth
from test_gpu_parity import check_case, pick_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tma", ["0", "1"])
@pytest.mark.parametrize("nx,ny,nz,fw,nmech,free_surf", [
    (11, 11, 11, 5, 0, 1),   # one interior cell an axis: both z faces in one row of words
    (9, 10, 15, 4, 0, 0),    # seven interior cells: the last width with whole z rows
    (13, 9, 16, 4, 1, 0),    # eight: the first with the far face packed
    (16, 17, 33, 3, 0, 1),   # a box of one cell along z
    (17, 13, 34, 6, 2, 1),
    (8, 23, 35, 3, 0, 0),    # a quad with one cell missing
    (25, 12, 64, 5, 3, 1),   # whole boxes along z
    (24, 33, 21, 10, 1, 1),  # a frame of ten, one interior cell along z
])
def test_edges_of_quads_and_boxes(tma, nx, ny, nz, fw, nmech, free_surf, oracle, request, monkeypatch):
    monkeypatch.setenv("IFOSB_TMA", tma)
    c = synth.small_case(nx=nx, ny=ny, nz=nz, fw=fw, nt=24, nmech=nmech, free_surf=free_surf, nshots=2, ntr=5, seed=nx + nz)
    check_case(c, pick_oracle(nmech, oracle, request))


@pytest.mark.parametrize("nt,ntast,nf", [(2, 1, 1), (8, 1, 2), (9, 1, 5), (17, 2, 3), (25, 3, 1), (10, 7, 4), (16, 1, 16)])
def test_dft_passes_of_every_length(nt, ntast, nf, oracle, request):
    c = synth.small_case(nx=19, ny=18, nz=23, nt=nt, nshots=2, seed=nt, finv=tuple(100.0 + 40.0 * q for q in range(nf)))
    c["ntast"] = ntast
    check_case(c, pick_oracle(0, oracle, request))


@pytest.mark.parametrize("tma", ["0", "1"])
@pytest.mark.parametrize("scale", [1e-30, 1e-36, 1e-42, 1e12, 1e22])
def test_quotients_of_every_magnitude(scale, tma, oracle, request, monkeypatch):
    """Sources from subnormal to beyond the fast division's dividends, spacing not a power of two."""
    monkeypatch.setenv("IFOSB_TMA", tma)
    c = synth.small_case(nx=21, ny=20, nz=27, nt=30, seed=7, finv=())
    c["params"].dx = c["params"].dy = c["params"].dz = np.float32(1.3)
    c["shots"][0][0, 5] = scale
    check_case(c, pick_oracle(0, oracle, request))


@pytest.mark.parametrize("rho", [3e-4, 4e7])
def test_densities_outside_the_fast_division(rho, oracle, request):
    c = synth.small_case(nx=18, ny=17, nz=22, nt=30, seed=9, finv=(300.0,))
    for w in ("true", "start"):
        vp, vs, r = c[w]
        c[w] = (vp, vs, (r / np.float32(2000.0) * np.float32(rho)).astype(np.float32))
    check_case(c, pick_oracle(0, oracle, request))
