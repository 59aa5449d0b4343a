"""The step-wise P2G adds up runs of neighbouring particles that share a cell
(csrc/k_stepwise.cuh): any order of the particles, block sizes that leave a
warp part empty and counts around a warp's edge give the oracle's result.

Tolerance: FP64 sums in another order, as the suite's other FP64 bars: 1e-9."""
import numpy as np
import pytest

import icempm_b200 as im

from mpm_cases import compare_states, gpu_model, gpu_state, oracle_run, params, scene


def _ordered(p, soa, order):
    """The same particles in another order (every row and the byte-packed
    crushed flags and grain ids)."""
    out = np.zeros_like(soa)
    S, T = im.SoA(soa, p.nPtsPitch, p.nPts), im.SoA(out, p.nPtsPitch, p.nPts)
    for name in ("P", "Q", "Jp_inv"):
        getattr(T, name)[:] = getattr(S, name)[order]
    for name in ("pos", "vel", "Fe", "Bp"):
        getattr(T, name)[:] = getattr(S, name)[:, order]
    T.crushed[:], T.grain[:] = S.crushed[order], S.grain[order]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("tpb", [256, 100, 33, 1])
@pytest.mark.parametrize("kind", ["sorted", "reversed", "shuffled", "interleaved", "one_cell"])
def test_any_order_and_block_size_matches_the_oracle(kind, tpb):
    p = params()
    p.tpb_P2G = tpb
    soa = scene(p, cells=(17, 7), seed=3, perturb=4e-4, vel=0.3, crushed_frac=0.1, jp_spread=1e-3)
    n = int(p.nPts)
    order = np.arange(n)
    if kind == "reversed":
        order = order[::-1].copy()
    elif kind == "shuffled":
        order = np.random.default_rng(1).permutation(n)
    elif kind == "interleaved":
        order = order.reshape(4, -1).T.reshape(-1).copy()
    soa = _ordered(p, soa, order)
    if kind == "one_cell":
        S = im.SoA(soa, p.nPtsPitch, p.nPts)
        S.pos[:, :45] = S.pos[:, :1]
    _, ref, _, _, _ = oracle_run(p, soa, 5)
    m = gpu_model(p, soa, im.FORM_FP64_STEPWISE)
    m.gpu.run_substeps(m.prms, 5)
    err = compare_states(p, gpu_state(m), ref, soa)
    m.gpu.close()
    assert err["disp_h"] <= 1e-9 and err["vel"] <= 1e-9 and err["strain"] <= 1e-9 and err["Bp"] <= 1e-9, err


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257])
@pytest.mark.parametrize("steps", [1, 2, 3])
def test_few_particles_and_the_grid_left_behind(n, steps):
    """The grid a run leaves is the last substep's, whichever of the two
    grids the run started on."""
    p = params()
    whole = scene(p, cells=(17, 7), seed=4, vel=0.2)
    pitch, p.nPts, p.nPtsPitch = int(p.nPtsPitch), n, im.pitch_elems(n)
    soa = np.zeros(im.N_PTS_ARRAYS * p.nPtsPitch)
    im.repitch_soa(whole, pitch, n, soa, int(p.nPtsPitch))
    _, ref, _, _, _ = oracle_run(p, soa, steps)
    a = gpu_model(p, soa, im.FORM_FP64_STEPWISE)
    a.gpu.run_substeps(a.prms, steps)
    err = compare_states(p, gpu_state(a), ref, soa)
    assert err["disp_h"] <= 1e-9 and err["vel"] <= 1e-9, err
    b = gpu_model(p, soa, im.FORM_FP64_STEPWISE)
    for k in range(steps):
        b.prms.SimulationTime += b.prms.InitialTimeStep
        b.gpu.cuda_reset_grid()
        b.gpu.cuda_p2g()
        b.gpu.cuda_update_nodes(b.prms.indenter_x_initial + b.prms.SimulationTime * b.prms.IndVelocity, b.prms.indenter_y)
        b.gpu.cuda_g2p(False)
    ga, gb = a.gpu.grid_from_device(), b.gpu.grid_from_device()
    assert np.abs(ga - gb).max() <= 1e-9 * np.abs(gb).max()
    a.gpu.close()
    b.gpu.close()
