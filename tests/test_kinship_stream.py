"""Streamed kinship: records kept on the device by pass 1 against records read twice, and the
.fam/.bim checks that stand for the full metadata."""

import numpy as np
import pytest

from jamma_b200 import io as jio
from jamma_b200 import kinship as kk


def _write(tmp_path, g):
    n, p = g.shape
    pre = tmp_path / "d"
    with open(f"{pre}.bed", "wb") as f:
        f.write(jio.BED_MAGIC)
        f.write(jio.pack_genotypes(g).tobytes())
    with open(f"{pre}.fam", "w") as f:
        f.writelines(f"f{i} s{i} 0 0 1 1.0\n" for i in range(n))
    with open(f"{pre}.bim", "w") as f:
        f.writelines(f"1\trs{j}\t0\t{j}\tA\tG\n" for j in range(p))
    return pre


@pytest.mark.parametrize("name,text", [
    ("fam", "f0 s0 0 0 1 1\nf1\n"), ("bim", "1 rs0 0 x A G\n"), ("bim", "1 rs0 0 5 A\n"),
    ("bim", "1 rs0 0 5 A\n1 rs1 0 x A G\n"),
])
def test_malformed_metadata_raises_the_same_error(tmp_path, name, text):
    pre = _write(tmp_path, np.zeros((2, 1)))
    assert jio.get_plink_dimensions(pre) == (2, 1)
    with open(f"{pre}.{name}", "w") as f:
        f.write(text)
    with pytest.raises((IndexError, ValueError)) as want:
        jio.get_plink_metadata(pre)
    with pytest.raises(want.type) as got:
        jio.BedFile(pre)
    assert str(got.value) == str(want.value)
    with pytest.raises(want.type) as late:
        jio.open_bed(pre)[1]()
    assert str(late.value) == str(want.value)


@pytest.mark.parametrize("bed_bytes,snps", [(1, 1), (4, 3), (5, 1), (0, 1)])
def test_size_mismatch_raises_the_same_error(tmp_path, bed_bytes, snps):
    pre = _write(tmp_path, np.zeros((3, snps)))
    with open(f"{pre}.bed", "wb") as f:
        f.write((jio.BED_MAGIC + bytes(4))[:3 + bed_bytes] if bed_bytes else b"\0\0\0\0")
    if snps == bed_bytes:
        assert jio.open_bed(pre)[1]() is None
        return
    with pytest.raises(ValueError) as want:
        jio.BedFile(pre)
    with pytest.raises(ValueError) as got:
        jio.open_bed(pre)[1]()
    assert str(got.value) == str(want.value)


def test_blank_lines_are_skipped(tmp_path):
    pre = _write(tmp_path, np.zeros((3, 2)))
    for name in ("fam", "bim"):
        with open(f"{pre}.{name}") as f:
            text = f.read()
        with open(f"{pre}.{name}", "w") as f:
            f.write("\n" + text.replace("\n", "\n \t\n"))
    assert jio.get_plink_dimensions(pre) == (3, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,mode", [("fp64", 1), ("int8", 1), ("fp64", 2)])
@pytest.mark.parametrize("subset", [False, True])
@pytest.mark.parametrize("maf", [0.0, 0.2])
def test_resident_and_reread_records_give_the_same_matrix(tmp_path, precision, mode, subset, maf,
                                                          monkeypatch):
    rng = np.random.default_rng(3)
    n, p = 203, 611
    g = rng.binomial(2, rng.uniform(0.05, 0.5, p), (n, p)).astype(np.float64)
    g[rng.random((n, p)) < 0.02] = np.nan
    pre = _write(tmp_path, g)
    sidx = np.arange(0, n, 2) if subset else None
    from jamma_b200 import engine as eng
    monkeypatch.setattr(eng, "READ_STAGE_BYTES", 51 * 100)  # pass 1 in pieces of 100 SNPs

    def run():
        return kk.compute_kinship_from_bed(pre, maf_threshold=maf, sample_idx=sidx,
                                           precision=precision, kinship_mode=mode)
    real = kk._selected_records
    monkeypatch.setattr(kk, "_selected_records", lambda b, i, s, kept: real(b, i, 150, kept))
    K = run()
    monkeypatch.setattr(kk, "_resident_records", lambda *a: None)
    assert np.array_equal(run(), K)
    X = g if sidx is None else g[sidx]
    X = X - np.nanmean(X, axis=0)
    af = np.nanmean(g if sidx is None else g[sidx], axis=0) / 2
    X = X[:, np.minimum(af, 1 - af) >= maf]
    if mode == 1:
        X = np.nan_to_num(X)
        assert np.max(np.abs(K - X @ X.T / X.shape[1])) <= 1e-13
