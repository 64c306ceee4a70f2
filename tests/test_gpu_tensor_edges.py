"""Tensor-core kernels at the edges of their tiles: every contingency table of a scan, as the kernel
that serves it computes them, against the oracle's (64-bit digests of all tables), and the top-N
against the full-table kernel's.  Sizes sit on and beside the tile edges of the kernels: 8 SNPs (column
groups), 64 and 120 SNPs (tiles), 64 and 256 samples (steps and stages of a class)."""
import pytest

pytestmark = pytest.mark.gpu

EDGES_3 = [  # snps, cases, controls
    (3, 1, 1), (9, 63, 64), (10, 65, 1), (65, 64, 257), (66, 256, 255), (67, 300, 129),
    (121, 512, 40), (130, 1023, 1025), (186, 100, 4000), (251, 2047, 2049), (129, 4095, 90),
]


def _data(snps, cases, ctrls, seed):
    from fiuncho_gb300 import Dataset, synth
    geno, is_case, _ = synth.simulate(synth.ScanSpec(snps, cases, ctrls, 3, 10, seed=seed))
    return Dataset.from_genotypes(geno, is_case)


def _check(order, snps, cases, ctrls, oracle, dist=None):
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    ds = _data(snps, cases, ctrls, 1000 * order + snps)
    gs = GpuSearch(0)
    res = Resident(gs.ctx, ds)
    d = dist or Distribution(snps, order - 1)
    got, count = gs.scan_digest(res, order, d, kernel=_lib.KERNEL_TENSOR)
    want = oracle.table_digest(ds.data, snps, ds.cases_words, ds.ctrls_words, order,
                               dist=(snps, d.step, d.offset))
    assert (got, count) == want
    gs.set_kernel(_lib.KERNEL_TENSOR)
    a = gs.run(res, order, d, 25)
    gs.set_kernel(_lib.KERNEL_FULL)
    b = gs.run(res, order, d, 25)
    assert [r.combination for r in a] == [r.combination for r in b]
    assert [r.val for r in a] == [r.val for r in b]


@pytest.mark.parametrize("snps,cases,ctrls", EDGES_3)
def test_order3_tile_edges(oracle, snps, cases, ctrls):
    _check(3, snps, cases, ctrls, oracle)


@pytest.mark.parametrize("snps,step,offset", [(70, 2, 1), (135, 3, 0), (66, 67, 5), (129, 5, 4)])
def test_order3_layer_edges(oracle, snps, step, offset):
    from fiuncho_gb300 import Distribution
    _check(3, snps, 130, 199, oracle, Distribution(snps, 2, step, offset))
