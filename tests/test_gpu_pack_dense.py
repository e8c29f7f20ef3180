"""Dense genotypes packed on the device against the host packing, byte for byte."""

import numpy as np
import pytest

from jamma_b200 import engine as eng
from jamma_b200.io import pack_genotypes


def _genotypes(n, p, dtype, order):
    rng = np.random.default_rng(n * 7 + p)
    g = rng.integers(0, 3, (n, p)).astype(dtype)
    if np.issubdtype(g.dtype, np.floating):
        g[rng.random((n, p)) < 0.03] = np.nan
        g[rng.random((n, p)) < 0.01] = -0.0
    return np.asarray(g, order=order)


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("n,p,dtype", [
    (1, 16384, np.float64), (16385, 1, np.float32), (127, 130, np.float64), (128, 129, np.float32),
    (130, 1001, np.float64), (1003, 333, np.float32), (515, 64, np.int8), (100, 20, np.float64),
])
def test_same_bytes_as_the_host_packing(n, p, dtype, order, monkeypatch):
    monkeypatch.setattr(eng, "PACK_STAGE_BYTES", 100_000)  # several pieces
    g = _genotypes(n, p, dtype, order)
    assert np.array_equal(eng.pack_on_device(g).cpu().numpy(), pack_genotypes(g))


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("bad", [0.5, 3.0, -1.0, np.inf, -np.inf])
def test_other_values_are_refused(bad, order):
    g = _genotypes(301, 77, np.float64, order)
    g[300, 76] = bad
    with pytest.raises(ValueError, match="allele counts 0/1/2 or NaN"):
        eng.pack_on_device(g)


@pytest.mark.gpu
def test_views_and_read_only_arrays():
    g = _genotypes(402, 300, np.float64, "C")
    v = g[::2]  # neither order: packed by the host
    assert np.array_equal(eng.pack_on_device(v).cpu().numpy(), pack_genotypes(v))
    g.setflags(write=False)
    assert np.array_equal(eng.pack_on_device(g).cpu().numpy(), pack_genotypes(g))
