"""The FP32 form lists a tile's nodes inside the indenter before a substep's
wait (csrc/k_pair32.cuh): tiles with no, few and only such nodes, indenters at
the grid's left wall and floor, one to sixteen warps a tile, split tiles,
against the CPU oracle.

Tolerance: a node's momentum is an FP32 sum of at most 36 terms (36 * 2^-24 =
2e-6 of their magnitude); the reaction is the part of it that the indenter
takes, here more than 1/100 of it, so 2e-4 a substep; 1e-3 of the largest for
two. Velocities: 1e-4 of their scale."""
import pytest

import icempm_b200 as im

from mpm_cases import compare_states, gpu_model, gpu_state, max_rel, oracle_run, params, scene


@pytest.mark.gpu
@pytest.mark.parametrize("tile,threads", [(0, 32), (1, 128), (1, 96), (2, 64), (3, 128)])
@pytest.mark.parametrize("diameter,x,y", [(0.02, 0.375, 0.08), (0.3, 0.375, 0.1), (0.1, 0.02, 0.03), (0.25, 0.3, 0.0)])
def test_reaction_matches_the_oracle(tile, threads, diameter, x, y):
    p = params(IndVelocity=0.5, IndDiameter=diameter)
    soa = scene(p, cells=(80, 16), seed=8, perturb=2e-4, vel=0.5)
    p.indenter_x = p.indenter_x_initial = x
    p.indenter_y = y
    n = 2
    _, ref, bins, _, hist = oracle_run(p, soa, n)
    m = gpu_model(p, soa, im.FORM_FP32, tile=tile, threads=threads)
    m.gpu.set_rebin_interval(1)  # the second substep splits the tiles the first found heavy
    m.gpu.set_tile_split(8, 0.5)
    m.gpu.run_substeps(m.prms, n)
    err = compare_states(p, gpu_state(m), ref, soa)
    assert m.gpu.error_code == 0 and bins.any()
    got, fh = m.gpu.host_side_indenter_force_accumulator.copy(), m.gpu.force_history(n)
    m.gpu.close()
    assert max_rel(got, bins) < 1e-3 and max_rel(fh, hist) < 1e-3
    assert err["vel"] <= 1e-4, err
