"""Paths of the engine that the common cases pass by, bit for bit against the oracle:
spacings that are no power of two in every kernel that divides by them, velocities and DFT
accumulators beyond the DFT pass's fast rounding, models handed over without ghost layers."""
import numpy as np
import pytest

import ifosb
import test_td_gradient_gpu
from helpers import engine_for, ifo_params
from ifosb import synth
from test_gpu_parity import check_case, pick_oracle

pytestmark = pytest.mark.gpu

small_case = synth.small_case


def spaced(**kw):
    c = small_case(**kw)
    p = c["params"]
    p.dx, p.dy, p.dz = np.float32(1.3), np.float32(1.1), np.float32(0.9)
    return c


@pytest.mark.parametrize("tma", ["0", "1"])
@pytest.mark.parametrize("nmech", [0, 1, 3, 4])
def test_gradient_at_other_spacings(nmech, tma, oracle, request, monkeypatch):
    monkeypatch.setenv("IFOSB_TMA", tma)
    c = spaced(nx=21, ny=18, nz=37, nt=40, nmech=nmech, nshots=2, seed=nmech + 50)
    check_case(c, pick_oracle(nmech, oracle, request))


@pytest.mark.parametrize("free_surf,interval,nmech", [(1, 3, 0), (0, 4, 3)])
def test_time_domain_kernels_at_other_spacings(oracle, free_surf, interval, nmech, monkeypatch):
    monkeypatch.setattr(synth, "small_case", spaced)
    test_td_gradient_gpu.test_time_domain_kernels_match_oracle_restatement(oracle, free_surf, interval, nmech)


def hess_f(p, rho, pi, u, finv, fwd, greens):
    """hess_F (hess_F.c:67-155) in float32: shots, then receivers, then frequencies."""
    b1, b2 = np.float32(1.1382), np.float32(-0.046414)
    two, four = np.float32(2.0), np.float32(4.0)
    h = np.zeros((3, p.ny, p.nx, p.nz), np.float32)
    inner = lambda a: test_td_gradient_gpu.interior(a, p)
    for F in fwd:
        for B in greens:
            for l, f in enumerate(finv):
                fd = np.float32(1.0) / np.float32(np.float64(f) * np.pi * 2)
                fr, fi, br, bi = ([x[c, l] for c in w] for x in (F, B) for w in ((0, 1, 2), (3, 4, 5)))
                (v, w, a, b) = (test_td_gradient_gpu.stencils(*x, p, b1, b2) for x in (fr, fi, br, bi))
                f6, b6 = [inner(x) for x in fr + fi], [inner(x) for x in br + bi]
                fdiv, fidiv, bdiv, bidiv = (x[0] + x[4] + x[8] for x in (v, w, a, b))
                relam = fd * (fidiv * bdiv + fdiv * bidiv)
                imlam = fd * (fidiv * bidiv - fdiv * bdiv)
                remu = (two * w[0] * a[0] + two * w[4] * a[4] + two * w[8] * a[8] + two * v[0] * b[0] + two * v[4] * b[4] +
                        two * v[8] * b[8] + (w[1] + w[3]) * (a[1] + a[3]) + (v[1] + v[3]) * (b[1] + b[3]) +
                        (w[2] + w[6]) * (a[2] + a[6]) + (v[2] + v[6]) * (b[2] + b[6]) + (w[5] + w[7]) * (a[5] + a[7]) +
                        (v[5] + v[7]) * (b[5] + b[7]))
                immu = (two * w[0] * b[0] + two * w[4] * b[4] + two * w[8] * b[8] - two * v[0] * a[0] - two * v[4] * a[4] -
                        two * v[8] * a[8] + (w[1] + w[3]) * (b[1] + b[3]) - (v[1] + v[3]) * (a[1] + a[3]) +
                        (w[2] + w[6]) * (b[2] + b[6]) - (v[2] + v[6]) * (a[2] + a[6]) + (w[5] + w[7]) * (b[5] + b[7]) -
                        (v[5] + v[7]) * (a[5] + a[7]))
                remu, immu = fd * remu, fd * immu
                dot = lambda x, y: x[0] * y[0] + x[1] * y[1] + x[2] * y[2]
                rerho = dot(f6[:3], b6[:3]) - dot(f6[3:], b6[3:])
                imrho = dot(f6[:3], b6[3:]) + dot(f6[3:], b6[:3])
                revs, imvs = -two * relam + remu, -two * imlam + immu
                rerho1 = rerho + relam * (pi - two * u) / rho + remu * u / rho
                imrho1 = imrho + imlam * (pi - two * u) / rho + immu * u / rho
                h[0] += (relam * relam + imlam * imlam) * rho * pi * four
                h[1] += (revs * revs + imvs * imvs) * four * rho * u
                h[2] += rerho1 * rerho1 + imrho1 * imrho1
    return h


@pytest.mark.parametrize("make", [small_case, spaced])
def test_hessian_against_a_restatement(make, oracle):
    c = make(nx=26, ny=22, nz=25, nt=60, fw=5, nshots=2, seed=31, free_surf=1)
    e, m, cp, shots = engine_for(c)
    p, q, rec = c["params"], ifo_params(c), np.asarray(c["recpos"], np.int32)
    sig = np.zeros((3, p.nt), np.float32)
    for r in range(3):
        sig[r, 5 + 4 * r:] = 1.0
    e.hessian_green([0, 1, 2], sig)
    e.zero_hessian()
    e.forward(shots, want_sections=False)
    e.hessian()
    greens = []
    for r in range(3):
        diff = np.zeros((3, 1, p.nt), np.float32)
        diff[1, 0] = sig[r]
        greens.append(oracle.adjoint(q, m, cp, rec[r:r + 1], diff, c["finv"], c["ntast"])["dft"])
    fwd = [oracle.forward(q, m, cp, sp, s, c["recpos"], c["finv"], c["ntast"], True)["dft"] for sp, s in shots]
    want = hess_f(p, *(m[k].reshape(p.ny, p.nx, p.nz) for k in ("rho", "pi", "u")), c["finv"], fwd, greens)
    assert np.isfinite(want).all() and all(np.abs(w).max() > 0 for w in want)
    assert np.array_equal(e.get_hessian(), want)
    e.close()


@pytest.mark.parametrize("tma", ["0", "1"])
def test_dft_of_huge_velocities(tma, oracle, monkeypatch):
    """An eighth of the velocities and a few accumulators above 2^100, all of them finite."""
    monkeypatch.setenv("IFOSB_TMA", tma)
    c = small_case(nx=19, ny=18, nz=23, nt=30, seed=7, free_surf=0)
    vp, vs, rho = c["start"]
    c["start"] = (vp, vs, rho * np.float32(1e-6))
    e, m, cp, ((sp, sig),) = engine_for(c)
    sig = (sig / np.abs(sig).max() * np.float32(1e35)).astype(np.float32)
    f = oracle.forward(ifo_params(c), m, cp, sp, sig, c["recpos"], c["finv"], 1, True, True)
    big = [np.abs(x) > 2.0**100 for x in (np.asarray(f["state"][:3]), f["dft"])]
    assert all(0 < b.mean() < 0.5 for b in big) and np.isfinite(f["dft"]).all()
    sec = e.forward([(sp, sig)])
    assert np.array_equal(sec[0], f["sections"])
    assert np.array_equal(e.get_dft(0), f["dft"])
    e.close()


def model_of(p, nmech, rng):
    shape = (p.ny, p.nx, p.nz)
    around = lambda x: (x * (1 + 0.1 * rng.random(shape))).astype(np.float32)
    m = [around(2000.0), around(1.8e10), around(6e9)]
    return m + ([around(0.05), around(0.04), np.linspace(0.01, 0.1, nmech, dtype=np.float32)] if nmech else [None] * 3)


@pytest.mark.parametrize("nx,ny,nz,nmech,nt", [
    (23, 21, 26, 0, 60),
    (24, 19, 25, 2, 60),      # relaxation times per cell
    (129, 128, 131, 0, 12),   # checked by several threads, copied through the chunks
])
def test_models_without_ghost_layers(nx, ny, nz, nmech, nt):
    c = small_case(nx=nx, ny=ny, nz=nz, nt=nt, nmech=nmech, nsrc=12, seed=nx)
    p, rng = c["params"], np.random.default_rng(nz)
    m = model_of(p, nmech, rng)
    e, _, _, shots = engine_for(c)
    ghost = [a if a is None or a.ndim == 1 else ifosb.ghost_wrap(a) for a in m]
    out = []
    for args, ghosted in ((m, False), (ghost, True)):
        e.set_model(*args, ghosted=ghosted)
        traces = e.forward(shots)
        out.append((traces, e.get_state(0), e.get_dft(0)))
    assert all(np.abs(a).max() > 0 for a in out[0][1:])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    # a bad cell is named in the ghosted order, whichever way the model comes, and the
    # model before stays
    e.set_model(*m)
    for q in range(3):
        for j, i, k in ((0, 0, 0), (ny - 1, nx - 1, nz - 1), (ny // 2, 3, nz - 2)):
            for value in (0.0, -1.0, np.inf, np.nan):
                bad = [None if a is None else a.copy() for a in m]
                bad[q][j, i, k] = value
                first = int(np.flatnonzero(~np.isfinite(ifosb.ghost_wrap(bad[q])) | (ifosb.ghost_wrap(bad[q]) <= 0))[0])
                said = []
                for args, ghosted in ((bad, False), ([a if a is None or a.ndim == 1 else ifosb.ghost_wrap(a) for a in bad], True)):
                    with pytest.raises(ifosb.IfosbError) as ei:
                        e.set_model(*args, ghosted=ghosted)
                    said.append(str(ei.value))
                assert said[0] == said[1] and said[0].endswith(f"ghosted index {first}")
                if nx > 100:
                    break
    assert np.array_equal(e.forward(shots), out[0][0])
    e.close()
