"""Tensor-core kernels at the edges of their tiles: every contingency table of a scan, as the kernel
that serves it computes them, against the oracle's (64-bit digests of all tables), and the top-N
against the full-table kernel's.  Sizes sit on and beside the tile edges of the kernels: 8 SNPs (column
groups), 16, 32 and 64 SNPs (rows of a tile), 112 and 120 SNPs (columns), 64 and 256 samples (steps and
stages of a class)."""
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


EDGES_4 = [  # snps, cases, controls
    (4, 1, 1), (5, 64, 65), (9, 63, 256), (17, 257, 129), (33, 65, 300), (34, 1023, 40), (36, 50, 4000),
    (47, 2047, 2049),
]


@pytest.mark.parametrize("snps,cases,ctrls", EDGES_4)
def test_order4_tile_edges(oracle, snps, cases, ctrls):
    _check(4, snps, cases, ctrls, oracle)


@pytest.mark.parametrize("snps,step,offset", [(20, 2, 1), (37, 3, 0), (18, 19, 5), (40, 5, 4)])
def test_order4_layer_edges(oracle, snps, step, offset):
    from fiuncho_gb300 import Distribution
    _check(4, snps, 130, 199, oracle, Distribution(snps, 3, step, offset))


SPLIT = [  # classes that do not share an accumulator: order, snps, cases, controls
    (3, 3, 4100, 4100), (3, 65, 9000, 9800), (3, 66, 4097, 4160), (3, 121, 300, 65000), (3, 130, 16384, 5000),
    (4, 4, 4100, 4100), (4, 33, 4097, 4160), (4, 36, 9000, 9800), (4, 19, 300, 65000),
]


@pytest.mark.parametrize("order,snps,cases,ctrls", SPLIT)
def test_split_classes_tile_edges(oracle, order, snps, cases, ctrls):
    from fiuncho_gb300 import GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    ds = _data(snps, cases, ctrls, 1000 * order + snps)
    gs = GpuSearch(0)
    res = Resident(gs.ctx, ds)
    assert gs.scan_digest(res, order, kernel=_lib.KERNEL_TENSOR) == \
        oracle.table_digest(ds.data, snps, ds.cases_words, ds.ctrls_words, order, dist=(snps, 1, 0))


@pytest.mark.parametrize("order,snps,step,offset", [(3, 70, 2, 1), (3, 135, 3, 0), (4, 37, 3, 0), (4, 20, 2, 1)])
def test_split_classes_layer_edges(oracle, order, snps, step, offset):
    from fiuncho_gb300 import Distribution
    _check(order, snps, 4100, 4101, oracle, Distribution(snps, order - 1, step, offset))


@pytest.mark.parametrize("snps,order", [(130, 4), (260, 3)])
def test_wide_tiles_against_the_reduced_work_kernel(snps, order):
    """Full column tiles (112 and 120 SNPs): digests of two kernels that share no code path."""
    from fiuncho_gb300 import GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    res = Resident(gs.ctx, _data(snps, 150, 201, 7 + snps))
    assert gs.scan_digest(res, order, kernel=_lib.KERNEL_TENSOR) == \
        gs.scan_digest(res, order, kernel=_lib.KERNEL_ELIDED_POPC)


@pytest.mark.parametrize("order,snps,outputs", [(3, 150, 1), (3, 150, 7000), (3, 40, 7000), (4, 60, 3), (4, 60, 7000),
                                                (4, 20, 7000)])
def test_threshold_raised_in_the_kernel_keeps_the_list(order, snps, outputs):
    """The list does not depend on when the device raises the threshold: few and many outputs, more
    outputs than combinations, against the full-table kernel's chunked search; shards merged too."""
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    res = Resident(gs.ctx, _data(snps, 311, 290, 40 + snps))
    gs.set_kernel(_lib.KERNEL_TENSOR)
    d = Distribution(snps, order - 1)
    a = gs.run(res, order, d, outputs)
    parts = [r for s in range(3) for r in gs.run_shard(res, order, s, 3, outputs)]
    gs.set_kernel(_lib.KERNEL_FULL)
    b = gs.run(res, order, d, outputs)
    assert [(r.combination, r.val) for r in a] == [(r.combination, r.val) for r in b]
    if outputs < 100:
        parts.sort(key=lambda r: (-r.val, r.combination))
        assert [r.val for r in parts[:outputs]] == [r.val for r in b]


EDGES_2 = [  # snps, cases, controls; the last four do not share an accumulator
    (2, 1, 1), (8, 64, 65), (9, 63, 256), (65, 257, 129), (121, 65, 300), (129, 1023, 40), (241, 2047, 2049),
    (2, 4100, 4100), (121, 9000, 9800), (130, 300, 65000), (250, 8000, 8000),
]


@pytest.mark.parametrize("snps,cases,ctrls", EDGES_2)
def test_order2_tile_edges(oracle, snps, cases, ctrls):
    _check(2, snps, cases, ctrls, oracle)


@pytest.mark.parametrize("snps,step,offset", [(130, 2, 1), (263, 3, 0), (66, 67, 5), (260, 5, 4)])
@pytest.mark.parametrize("cases,ctrls", [(130, 199), (4100, 4101)])
def test_order2_layer_edges(oracle, snps, step, offset, cases, ctrls):
    from fiuncho_gb300 import Distribution
    _check(2, snps, cases, ctrls, oracle, Distribution(snps, 1, step, offset))


@pytest.mark.parametrize("order,snps,cases,ctrls", [(2, 1900, 4100, 4100), (2, 2100, 300, 290),
                                                    (3, 300, 4097, 4100), (4, 130, 4097, 4100)])
def test_several_items_per_pair(order, snps, cases, ctrls):
    """More items than CTA pairs, so that accumulators, stashes and tables are used again: every table and
    the list against a kernel that shares no code path."""
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    res = Resident(gs.ctx, _data(snps, cases, ctrls, 3 * snps))
    assert gs.scan_digest(res, order, kernel=_lib.KERNEL_TENSOR) == \
        gs.scan_digest(res, order, kernel=_lib.KERNEL_ELIDED_HS)
    lists = []
    for kernel in (_lib.KERNEL_TENSOR, _lib.KERNEL_ELIDED_HS):
        gs.set_kernel(kernel)
        lists.append([(r.combination, r.val) for r in gs.run(res, order, Distribution(snps, order - 1), 1000)])
    assert lists[0] == lists[1]


MISSING_3 = [  # snps, cases, controls, missing rate
    (32, 1, 1, 0.3), (33, 64, 65, 0.2), (41, 63, 256, 0.05), (65, 257, 129, 0.01), (66, 100, 300, 0.1),
    (97, 512, 40, 0.03), (130, 1023, 1025, 0.002), (177, 2047, 2049, 0.02), (121, 100, 4000, 0.5),
]


@pytest.mark.parametrize("snps,cases,ctrls,rate", MISSING_3)
def test_order3_missing_calls(snps, cases, ctrls, rate):
    """Data with missing calls: the list, for few outputs (a tight threshold) and for many, of the kernel that
    counts all 27 cells on the tensor cores against the full-table kernel's, and its shards'."""
    import numpy as np
    from fiuncho_gb300 import Dataset, Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    full = _data(snps, cases, ctrls, 5 * snps)
    rng = np.random.default_rng(snps)
    rows = full.data.copy().reshape(snps, -1)
    for at, words in ((0, full.cases_words), (3 * full.cases_words, full.ctrls_words)):
        called = np.packbits(rng.random((snps, 64 * words)) >= rate, axis=1, bitorder="little").view(np.uint64)
        for g in range(3):
            rows[:, at + g * words:at + (g + 1) * words] &= called
    ds = Dataset(cases, ctrls, snps, full.cases_words, full.ctrls_words, rows.reshape(-1))
    gs = GpuSearch(0)
    res = Resident(gs.ctx, ds)
    d = Distribution(snps, 2)
    for outputs in (3, 40, 3000):
        gs.set_kernel(_lib.KERNEL_AUTO)
        a = gs.run(res, 3, d, outputs)
        assert gs.last_tile()[0] == _lib.KERNEL_TENSOR
        parts = [r for s in range(3) for r in gs.run_shard(res, 3, s, 3, outputs)]
        gs.set_kernel(_lib.KERNEL_FULL)
        b = gs.run(res, 3, d, outputs)
        assert [(r.combination, r.val) for r in a] == [(r.combination, r.val) for r in b]
        parts.sort(key=lambda r: (-r.val, r.combination))
        assert [r.val for r in parts[:outputs]] == [r.val for r in b]


def test_order3_rows_that_share_samples_keep_the_full_tables():
    """Rows that are not genotypes (a sample in two of them, bits past the class) stay with the full-table
    kernel, which takes any data."""
    import numpy as np
    from fiuncho_gb300 import Dataset, Distribution, GpuSearch, _lib
    full = _data(40, 100, 90, 3)
    gs = GpuSearch(0)
    for change in ("shared", "past"):
        rows = full.data.copy().reshape(40, -1)
        if change == "shared":
            rows[7, 0] |= np.uint64(1)
            rows[7, full.cases_words] |= np.uint64(1)
        else:
            rows[7, full.cases_words - 1] |= np.uint64(1) << np.uint64(63)
        gs.run(Dataset(100, 90, 40, full.cases_words, full.ctrls_words, rows.reshape(-1)), 3, Distribution(40, 2), 5)
        assert gs.last_tile()[0] == _lib.KERNEL_FULL


@pytest.mark.parametrize("order,snps,step,offset", [
    (2, 130, 16_900_001, 0), (2, 260, 2 ** 28, 129), (2, 66, 2 ** 31 - 1, 5), (3, 70, 2 ** 28, 3),
    (3, 66, 2 ** 31 - 1, 64), (4, 40, 70_000_001, 0), (4, 37, 2 ** 28, 40), (4, 36, 2 ** 31 - 1, 7)])
def test_layers_of_steps_past_32_bit_positions(oracle, order, snps, step, offset):
    """A step so large that a tile's later positions would leave 32 bits owns one prefix, the one of rank
    `offset`: its tables and its list."""
    import math
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    ds = _data(snps, 300, 311, 90 + snps)
    gs = GpuSearch(0)
    res = Resident(gs.ctx, ds)
    d = Distribution(snps, order - 1, step, offset)
    digest, count = gs.scan_digest(res, order, d, kernel=_lib.KERNEL_TENSOR)
    assert (digest, count) == oracle.table_digest(ds.data, snps, ds.cases_words, ds.ctrls_words, order,
                                                  dist=(snps, math.comb(snps, order - 1), offset))
    lists = []
    for kernel in (_lib.KERNEL_AUTO, _lib.KERNEL_FULL):
        gs.set_kernel(kernel)
        lists.append([(r.combination, r.val) for r in gs.run(res, order, d, 25)])
    assert lists[0] == lists[1] and len(lists[0]) == min(25, count)


@pytest.mark.parametrize("snps,cases,ctrls,kernel", [(31, 300, 300, 2), (32, 300, 300, 4), (31, 600, 424, 4)])
def test_order4_choice_is_one_for_searches_batches_and_digests(snps, cases, ctrls, kernel):
    """The automatic order-4 kernel from 32 SNPs or 1 024 samples, below and above; a batch's lanes and the
    digest's own choice give what a search alone gives."""
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    res = Resident(gs.ctx, _data(snps, cases, ctrls, 60 + snps))
    d = Distribution(snps, 3)
    alone = gs.run(res, 4, d, 30)
    assert gs.last_tile()[0] == kernel
    (batched, _), = gs.run_batch([(res, 4, d, 30)])
    assert [(r.combination, r.val) for r in batched] == [(r.combination, r.val) for r in alone]
    assert gs.scan_digest(res, 4) == gs.scan_digest(res, 4, kernel=_lib.KERNEL_FULL)


@pytest.mark.parametrize("snps,cases,ctrls,step", [
    (60, 30, 900, 1), (60, 900, 30, 1), (50, 200, 7800, 1), (50, 7800, 200, 1), (45, 1000, 20000, 1),
    (45, 20000, 1000, 1), (40, 600, 60000, 1), (40, 60000, 600, 1), (60, 100, 3000, 3), (45, 1000, 20000, 2)])
def test_order4_uneven_classes(snps, cases, ctrls, step):
    """Classes of which one is many times the other: the bound rejects little there, and the estimate that
    follows it decides what gets an exact key.  Few outputs (a tight threshold) and many, against the
    full-table kernel."""
    from fiuncho_gb300 import Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    res = Resident(gs.ctx, _data(snps, cases, ctrls, 70 + snps))
    d = Distribution(snps, 3, step, step - 1)
    for outputs in (10, 3000):
        gs.set_kernel(_lib.KERNEL_TENSOR)
        a = gs.run(res, 4, d, outputs)
        gs.set_kernel(_lib.KERNEL_FULL)
        b = gs.run(res, 4, d, outputs)
        assert [(r.combination, r.val) for r in a] == [(r.combination, r.val) for r in b]


def test_order4_uneven_classes_cost_no_exact_key_each():
    """100 SNPs x 1 000 cases and 20 000 controls, where seven combinations in ten pass the bound, within five
    times the time of even classes (with an exact key for each of them 150 SNPs took 643 ms, now 16)."""
    import time
    from fiuncho_gb300 import Distribution, GpuSearch
    from fiuncho_gb300.search import Resident
    gs = GpuSearch(0)
    best = []
    for cases, ctrls in ((10500, 10500), (1000, 20000)):
        res = Resident(gs.ctx, _data(100, cases, ctrls, 71))
        times = []
        for _ in range(4):
            t = time.perf_counter()
            gs.run(res, 4, Distribution(100, 3), 50)
            times.append(time.perf_counter() - t)
        best.append(min(times))
    assert best[1] < 5 * best[0], best


@pytest.mark.parametrize("cases,ctrls", [(300, 311), (4100, 4101), (9000, 9800)])
@pytest.mark.parametrize("copies", [1, 8, 40])
def test_order4_many_keys_in_a_group(cases, ctrls, copies):
    """Groups of which several combinations reach the threshold -- SNPs that are copies of one another, and a
    layer whose first launch holds fewer combinations than are kept -- take all their keys at once: the
    lists against the full-table kernel's."""
    from fiuncho_gb300 import Dataset, Distribution, GpuSearch, _lib
    from fiuncho_gb300.search import Resident
    ds = _data(40, cases, ctrls, 72)
    rows = ds.data.copy().reshape(40, -1)
    rows[:copies] = rows[0]
    gs = GpuSearch(0)
    res = Resident(gs.ctx, Dataset(cases, ctrls, 40, ds.cases_words, ds.ctrls_words, rows.reshape(-1)))
    for step, outputs in ((1, 10), (1, 5000), (3, 7000)):
        d = Distribution(40, 3, step, step - 1)
        gs.set_kernel(_lib.KERNEL_TENSOR)
        a = gs.run(res, 4, d, outputs)
        gs.set_kernel(_lib.KERNEL_FULL)
        b = gs.run(res, 4, d, outputs)
        assert [(r.combination, r.val) for r in a] == [(r.combination, r.val) for r in b]


@pytest.mark.parametrize("cases,ctrls", [(300, 311), (4100, 4101)])
def test_order4_more_ties_than_the_buffer_holds(cases, ctrls):
    """916 895 combinations of equal value: the launch overflows its candidate buffer and is made again in
    pieces; the list is the first combinations'."""
    import itertools
    from fiuncho_gb300 import Dataset, Distribution, GpuSearch
    ds = _data(70, cases, ctrls, 73)
    rows = ds.data.copy().reshape(70, -1)
    rows[:] = rows[0]
    gs = GpuSearch(0)
    got = gs.run(Dataset(cases, ctrls, 70, ds.cases_words, ds.ctrls_words, rows.reshape(-1)), 4, Distribution(70, 3), 40)
    assert gs.last_tile()[0] == 4
    assert [tuple(r.combination) for r in got] == list(itertools.islice(itertools.combinations(range(70), 4), 40))


@pytest.mark.parametrize("i,j,l", [(0, 1, 2), (0, 63, 71), (3, 40, 41), (5, 70, 71), (7, 36, 69), (69, 70, 71)])
def test_order3_missing_calls_every_cell(i, j, l):
    """A combination whose association lies in one of its 27 cells, for every cell as the kernel for data with
    missing calls counts them (places at the edges of its tiles and halves): the best combinations (it and
    those that share two of its SNPs) against the full-table kernel's."""
    import itertools
    import numpy as np
    from fiuncho_gb300 import Dataset, Distribution, GpuSearch, _lib
    gs = GpuSearch(0)
    rng = np.random.default_rng(100 * i + j)
    base = rng.integers(0, 3, (72, 590)).astype(np.uint8)
    base[rng.random(base.shape) < 0.05] = 3
    is_case = np.arange(590) < 300
    for cell in itertools.product(range(3), repeat=3):
        geno = base.copy()
        rows = geno[[i, j, l]]
        rows[:, rng.choice(300, 50, replace=False)] = np.array(cell, np.uint8)[:, None]
        hit = (rows == np.array(cell, np.uint8)[:, None]).all(0) & ~is_case
        rows[rng.integers(0, 3), hit] = 3  # no control has it
        geno[[i, j, l]] = rows
        ds, lists = Dataset.from_genotypes(geno, is_case), []
        for kernel in (_lib.KERNEL_AUTO, _lib.KERNEL_FULL):
            gs.set_kernel(kernel)
            lists.append([(tuple(r.combination), r.val) for r in gs.run(ds, 3, Distribution(72, 2), 100)])
            assert gs.last_tile()[0] == (kernel or _lib.KERNEL_TENSOR)
        assert lists[0] == lists[1] and (i, j, l) in [c for c, _ in lists[0]], cell
