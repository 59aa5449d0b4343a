"""Full substeps of few tiles run with more threads than asked for (two to
eight warps in FP64, up to sixteen in FP32): a run that takes them, and one
context that changes form, block size and tile size between runs of the same
scene, against the CPU oracle."""
import pytest

import icempm_b200 as im

from mpm_cases import compare_states, gpu_model, gpu_state, oracle_run, params, scene


@pytest.mark.gpu
@pytest.mark.parametrize("tile,threads", [(0, 32), (0, 64), (1, 64), (1, 128), (2, 96), (3, 128)])
def test_fp64_few_tiles_match_the_oracle(tile, threads):
    """Sums of another order only: 64-bit rounding of 9 nodes' terms over 6
    substeps, below 1e-12 of each field's scale; 1e-9 leaves room for what the
    return mapping makes of it."""
    p = params()
    soa = scene(p, cells=(40, 20), seed=4, perturb=3e-4, vel=0.5, crushed_frac=0.2, jp_spread=2e-3)
    n = 6
    _, ref, _, _, _ = oracle_run(p, soa, n)
    m = gpu_model(p, soa, im.FORM_FP64, tile=tile, threads=threads)
    m.gpu.run_substeps(m.prms, n)
    err = compare_states(p, gpu_state(m), ref, soa)
    assert m.gpu.error_code == 0
    m.gpu.close()
    for k in ("disp_h", "vel", "strain"):
        assert err[k] <= 1e-9, (k, err)
    assert err["crushed_mismatch"] == 0, err


@pytest.mark.gpu
def test_one_context_changes_form_and_block():
    p = params()
    soa = scene(p, cells=(40, 20), seed=6, perturb=3e-4, vel=0.5)
    _, ref, _, _, _ = oracle_run(p, soa, 4)
    m = gpu_model(p, soa, im.FORM_FP32, tile=1, threads=128)
    for form, tile, threads in ((im.FORM_FP32, 1, 128), (im.FORM_FP64, 1, 128), (im.FORM_FP32, 1, 128),
                                (im.FORM_FP64, 0, 64), (im.FORM_FP32, 0, 64), (im.FORM_FP64, 1, 64)):
        m.gpu.set_form(form)
        m.gpu.set_tile(tile, threads)
        m.prms = p.copy()
        m.gpu.tmp_transfer_buffer[: soa.size] = soa
        m.gpu.transfer_ponts_to_device()
        m.gpu.run_substeps(m.prms, 4)
        err = compare_states(p, gpu_state(m), ref, soa)
        assert m.gpu.error_code == 0
        # FP32: as the pair loop's test; FP64: as above
        tol = 1e-4 if form == im.FORM_FP32 else 1e-9
        assert all(err[k] <= tol for k in ("disp_h", "vel", "strain")), (form, tile, threads, err)
    m.gpu.close()
