"""compute_kinship_from_bed's chunk_size bounds the SNPs decoded at a time on the device."""

import numpy as np
import pytest
from test_kinship_stream import _write

from jamma_b200 import kinship as kk


def test_device_chunk():
    assert [kk._device_chunk(c) for c in (1, 700, 9999, 10_000, 16_384, 20_000)] == \
        [1, 700, 9999, 16_384, 16_384, 20_000]


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,precision,mode", [(203, 1500, "fp64", 1), (203, 1500, "fp64", 2),
                                                (203, 1500, "int8", 1), (1100, 9000, "fp64", 1)])
@pytest.mark.parametrize("resident", [True, False])
def test_a_small_chunk_size_is_kept(tmp_path, n, p, precision, mode, resident, monkeypatch):
    rng = np.random.default_rng(n)
    g = rng.binomial(2, rng.uniform(0.05, 0.5, p), (n, p)).astype(np.float64)
    g[rng.random((n, p)) < 0.01] = np.nan
    pre = _write(tmp_path, g)
    want = kk.compute_kinship_from_bed(pre, precision=precision, kinship_mode=mode)
    if not resident:
        monkeypatch.setattr(kk, "_resident_records", lambda *a: None)
    rows, spaces = [], []
    decode, space = kk.decode_packed, kk.workspace
    monkeypatch.setattr(kk, "decode_packed", lambda r, *a: rows.append(r.shape[0]) or decode(r, *a))
    monkeypatch.setattr(kk, "workspace", lambda b: spaces.append(b) or space(b))
    K = kk.compute_kinship_from_bed(pre, chunk_size=350, precision=precision, kinship_mode=mode)
    assert max(rows) == 350
    assert max(spaces) < 350 * n * 8 + 64 * n * 8 + (1 << 20)
    # the same sums in other chunks: the rounding of p terms of at most 4
    assert np.abs(K - want).max() <= 1e-13 * np.abs(want).max() + 1e-12 * (mode == 2)
