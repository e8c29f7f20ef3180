"""The FP64 form's rotation of calls outside the ordinary chunk: no SNPs at all."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
def test_no_snps_give_empty_results(mode):
    import torch

    from jamma_b200 import engine as eng

    n = 64
    rng = np.random.default_rng(mode)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    cohort = eng.DeviceCohort(np.arange(n) / n, q, None, rng.standard_normal((n, 2)), mode)
    codes = torch.empty((0, cohort.code_ld), dtype=torch.int8, device="cuda")
    out = cohort.associate_codes(codes, torch.empty(0, dtype=torch.float64, device="cuda"))
    assert {k: tuple(v.shape) for k, v in out.items()} == {k: (2, 0) for k in eng.MODE_KEYS[mode]}
    assert cohort.rotate_status() == 0
