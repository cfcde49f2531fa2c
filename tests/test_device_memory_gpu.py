"""Calls that need device memory while an engine holds its velocity ring, which it takes
from memory that is free and needs for speed alone: the ring makes way, the call works as
on an empty device, and the engine's later calls give the same bits without it."""
import contextlib

import numpy as np
import pytest

import ifosb
from helpers import engine_for
from ifosb import synth
from test_gpu_parity import check_case, pick_oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20
NX, NY, NZ, NT, SHOTS = 64, 56, 60, 24, 40
PZ = (NZ + 10 + 7) // 8 * 8
FIELD = (NY + 5) * (NX + 4) * PZ  # floats of a field with its halos
RING = 7 * 3 * FIELD * 4 * SHOTS


@contextlib.contextmanager
def little_memory(leave):
    """All of the device's free memory but `leave` bytes taken by somebody else."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del taken
        torch.cuda.empty_cache()


def engine_with_ring(free_surf):
    """An engine that has run a forward with frequencies and holds the whole ring."""
    c = synth.small_case(nx=NX, ny=NY, nz=NZ, nt=NT, free_surf=free_surf, nshots=1, ntr=7, seed=4, finv=(300.0,))
    e, _, _, shots = engine_for(c, max_shots=SHOTS)
    before = e.device_bytes
    traces = e.forward(shots)
    assert e.device_bytes - before >= RING, "no ring to give back"
    e.residual((traces * np.float32(0.9)).astype(np.float32))
    return e, shots, traces


@pytest.mark.parametrize("free_surf", [0, 1])
def test_exact_vjp_takes_the_ring(free_surf):
    e, shots, traces = engine_with_ring(free_surf)
    dft = e.get_dft(0)
    want, want_mis = e.vjp_exact(12, moduli=True)
    held = e.device_bytes
    # 2 checkpoints, 13 states of a segment and the adjoint's, of 9 fields and their PML
    # memories in double: more than is free, less than that and the ring
    with little_memory(16 * 9 * FIELD * 8):
        got, mis = e.vjp_exact(12, moduli=True)
    assert e.device_bytes <= held - RING
    assert np.array_equal(got, want) and np.array_equal(mis, want_mis)
    assert np.array_equal(e.forward(shots), traces)
    assert np.array_equal(e.get_dft(0), dft), "DFT fields without the ring"
    e.close()


@pytest.mark.parametrize("what", ["engine", "optimiser"])
def test_other_objects_take_the_ring(what):
    e, shots, traces = engine_with_ring(1)
    dft, held = e.get_dft(0), e.device_bytes
    p = e.p
    with little_memory(RING // 2):  # more than is free, less than that and the ring
        if what == "engine":  # the wavefields alone, at 9 fields a shot
            other = ifosb.Engine(p, max_shots=RING * 3 // 4 // (9 * FIELD * 4), max_nf=0)
        else:  # two FP64 histories of two parameters
            other = ifosb.Optimizer(NX, NY, NZ, numpar=2, bfgsnum=RING * 3 // 4 // (2 * 2 * 8 * NX * NY * NZ))
        assert e.device_bytes == held - RING
        other.close()
    assert np.array_equal(e.forward(shots), traces)
    assert np.array_equal(e.get_dft(0), dft), "DFT fields without the ring"
    e.close()


@pytest.mark.parametrize("slots", [0, 1, 2, 6])
def test_a_capped_ring_changes_no_bit(slots, oracle, request, monkeypatch):
    monkeypatch.setenv("IFOSB_DFT_SLOTS", str(slots))
    c = synth.small_case(nx=19, ny=18, nz=23, nt=25, nshots=2, seed=slots)
    e, _ = check_case(c, pick_oracle(0, oracle, request))
    assert e.launch_count == 2 * 25 + -(-25 // (slots + 1)), "passes of slots + 1 DFT steps"
    e.close()
