"""A tensor-core rotation whose bounded wait ran out is reported however many rotations follow
it: by the cohort, by the association runner (before the chunk's results go anywhere) and by
the server.

As in test_gpu_bounded_wait.py the library's test hook shortens the deadline to 10 ms and turns
the tile loads off, so that the first wait runs out with no copy and no MMA in flight."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hook(on: bool) -> None:
    from jamma_b200 import _native

    if on:
        _native.call("jb_test_pipeline_timeout", 1, 10_000_000)
    else:
        _native.call("jb_test_pipeline_timeout", 0, 2_000_000_000)


@pytest.fixture
def one_cta_kernel():
    """The one-CTA rotation kernel carries the hook."""
    from jamma_b200 import _native

    prev = _native.load().jb_rotate_get_kernel()
    _native.call("jb_rotate_set_kernel", 0)
    yield
    _hook(False)
    _native.call("jb_rotate_set_kernel", prev)


def _cohort(precision, n=500, p=700):
    from jamma_b200 import engine as eng
    from jamma_b200 import synth
    from oracle import plink as OP

    g = synth.genotypes(n, p, 0.02, seed=5)
    ev, q = np.linalg.eigh(np.corrcoef(np.nan_to_num(g, nan=1.0)))
    y = np.random.default_rng(0).normal(size=n)
    cohort = eng.DeviceCohort(np.maximum(ev, 0.0), q, None, y, lmm_mode=1, precision=precision)
    return cohort, OP.encode_genotypes(g), np.nanmean(g, 0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("missing", [True, False])
def test_a_failed_rotation_is_told_after_later_ones(precision, missing, one_cta_kernel):
    import torch

    from jamma_b200 import engine as eng

    cohort, packed, mean = _cohort(precision)
    codes, _ = eng.decode_packed(torch.from_numpy(packed).cuda(), cohort.n, None, cohort.n, cohort.code_ld)
    if not missing:
        codes = torch.where(codes == 3, 0, codes).contiguous()
    mu = torch.from_numpy(mean).cuda()

    def rotate(rows):
        if precision == "mixed":
            return cohort.rotate_codes_i8(codes[:rows], mu[:rows], missing)
        return cohort.rotate_codes_f64(codes[:rows], mu[:rows], missing)

    good = rotate(200).clone()
    assert cohort.rotate_status() == 0
    _hook(True)
    rotate(200)
    _hook(False)
    rotate(200)
    rotate(700)  # a larger workspace keeps the report
    assert 100 < cohort.rotate_status() < 200
    assert cohort.rotate_status() == 0  # told once
    assert torch.equal(rotate(200), good)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_runner_raises_for_a_chunk_that_is_not_the_last(precision, one_cta_kernel):
    from jamma_b200.lmm import associate_records

    cohort, packed, mean = _cohort(precision)
    seen = []

    def records(s, e, out):
        _hook(s == 0)  # waits for the device: every chunk before this one has run
        out[:] = packed[s:e]

    with pytest.raises(RuntimeError, match="pipeline"):
        associate_records(cohort, records, cohort.n, None, mean, device_chunk=256,
                          on_chunk=lambda s, e: seen.append(s))
    assert seen == []
    res = associate_records(cohort, packed, cohort.n, None, mean, device_chunk=256)
    assert np.isfinite(res["p_wald"]).any()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_server_raises_and_goes_on(precision, one_cta_kernel):
    from jamma_b200 import synth
    from jamma_b200.serve import GwasJob, GwasServer
    from oracle import plink as OP

    n = 300
    g = synth.genotypes(n, 1200, 0.01, seed=400)
    packed = OP.encode_genotypes(g)
    y = np.random.default_rng(1).normal(size=n)
    srv = GwasServer(hbm_budget_bytes=8 << 30, max_active=1, chunk=256, precision=precision)
    srv.submit(GwasJob("bad", "A", packed, n, y, None, 1))
    while not srv.active:
        srv.step()
    act = srv.active[0]
    _hook(True)
    srv._launch_chunk(act)
    _hook(False)
    with pytest.raises(RuntimeError, match="bad"):
        while srv.active:
            srv.step()
    assert not srv.active and srv.used == 0 and srv.cohorts["A"].refs == 0
    srv.submit(GwasJob("good", "A", packed, n, y, None, 1))
    done = srv.run()
    assert [j.job_id for j in done] == ["good"]
    assert np.isfinite(done[0].results["p_wald"]).all()
