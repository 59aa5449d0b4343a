"""The FP32 form's full substep walks the particles of a cell in pairs, with
one to sixteen warps per tile (csrc/k_pair32.cuh): cells with odd counts and
none, cells beyond the pairs that one walk covers, particles that left their
cell, tiles run by more warps than they have groups of cells, and tiles whose
groups are split over two CTAs, each against the CPU oracle.

Tolerance: an FP32 sum of the densest cell's 300 particles carries at most
300 * 2^-24 = 2e-5 of its terms' magnitude, over three substeps 6e-5; 1e-4 of
each field's scale."""
import numpy as np
import pytest

import icempm_b200 as im

from mpm_cases import compare_states, gpu_model, gpu_state, oracle_run, params, scene


def _crowded(p, seed=5):
    """A block whose first particles are moved into a few cells: 1, 2, 3, 64,
    65, 140 and 300 of them, beside the lattice's 4 per cell."""
    soa = scene(p, cells=(40, 16), seed=seed, perturb=3e-4, vel=0.5, crushed_frac=0.2, jp_spread=2e-3)
    S = im.SoA(soa, p.nPtsPitch, p.nPts)
    rng = np.random.default_rng(seed)
    h, at = p.cellsize, 0
    for k, n in enumerate((1, 2, 3, 64, 65, 140, 300)):
        S.pos[0, at: at + n] = (70 + 3 * k % 20 + 0.5 + rng.random(n)) * h
        S.pos[1, at: at + n] = (20 + 3 * (k % 3) + 0.5 + rng.random(n)) * h
        at += n
    return soa


@pytest.mark.gpu
@pytest.mark.parametrize("tile,threads", [(0, 32), (0, 128), (1, 96), (1, 128), (1, 256), (2, 64), (3, 160), (3, 128)])
@pytest.mark.parametrize("rebin", [0, 2])
def test_crowded_and_odd_cells_match_the_oracle(tile, threads, rebin):
    p = params()
    soa = _crowded(p)
    n = 3
    _, ref, _, _, rh = oracle_run(p, soa, n)
    m = gpu_model(p, soa, im.FORM_FP32, tile=tile, threads=threads)
    m.gpu.set_rebin_interval(rebin)
    m.gpu.run_substeps(m.prms, n)
    err = compare_states(p, gpu_state(m), ref, soa)
    assert m.gpu.error_code == 0
    m.gpu.close()
    for k in ("disp_h", "vel", "strain"):
        assert err[k] <= 1e-4, (k, err)
    assert err["crushed_mismatch"] == 0, err


@pytest.mark.gpu
@pytest.mark.parametrize("form,tol", [(im.FORM_FP32, 1e-4), (im.FORM_FP64, 1e-9)])
def test_particles_far_from_their_cells_match_the_oracle(form, tol):
    """A fast block without re-binning: particles gather and scatter outside
    their cells, beyond their tile's region and across tiles."""
    p = params(IndVelocity=1.0)
    soa = scene(p, cells=(40, 12), seed=9, perturb=2e-4)
    im.SoA(soa, p.nPtsPitch, p.nPts).vel[0] = 400.0
    n = 40  # 4 cells of travel
    _, ref, _, _, _ = oracle_run(p, soa, n)
    m = gpu_model(p, soa, form, tile=1, threads=128)
    m.gpu.set_rebin_interval(0)
    m.gpu.run_substeps(m.prms, n)
    err = compare_states(p, gpu_state(m), ref, soa)
    strays = m.gpu.stray_count()
    m.gpu.close()
    assert strays > p.nPts
    assert err["disp_rel"] <= tol and err["vel"] <= tol, err
