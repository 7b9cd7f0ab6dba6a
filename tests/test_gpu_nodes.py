"""Pairs on frequency nodes (kg_node.cu) against the oracle, at the sizes where
the tiles can go wrong: one sample, sample counts around the 128-row tile, site
counts around the padded bins, a narrow and a wide range of frequencies, a
chunk boundary inside a row, a pair without a common site.

The objective's bar: the interpolation error of log d is below 2e-10 of a
site's term (FP32C's eight nodes a bin) and the fixed-point weights add less than
2^-30, averaged over the pair's sites, on an objective of order 1, and the two
sides stop within a KKT residual of 1e-8 of the same optimum, where the
objective differs by its square: 1e-9 relative holds with a margin.  Delta and
kinship keep the shared bar."""
import numpy as np
import pytest

import kestrel_b200 as kb
from kestrel_b200 import synth

from .parity import compare

pytestmark = pytest.mark.gpu

OBJ = 1e-9


def cohort(n, m, seed, missing=0.02):
    return synth.make_cohort(n, m, seed, missing=missing).codes


def check(est, codes, ref, **kw):
    est.load(codes, kw.pop("af", None))
    rows = est.relatedness(**kw)
    st = est.run_stats()
    assert st["fp64_passes"] == st["gh_passes"] > 0, "the cohort should run on nodes"
    print(compare(rows, ref))
    assert (np.abs(rows["obj"] - ref["obj"]) / np.abs(ref["obj"])).max() <= OBJ
    return rows


@pytest.mark.parametrize("n,m", [(1, 16_000), (2, 15_500), (31, 16_385), (129, 16_001)])
def test_sizes(oracle, n, m):
    codes = cohort(n, m, 700 + n)
    with kb.Estimator() as est:
        check(est, codes, oracle.relatedness(codes))


@pytest.mark.parametrize("spread", ["half", "wide", "edges"])
def test_frequencies(oracle, spread):
    n, m = 12, 40_000
    rng = np.random.default_rng(5)
    p = {"half": np.full(m, 0.5),
         "wide": np.exp(rng.uniform(np.log(2e-4), np.log(0.5), m)),
         "edges": 0.5 * 2.0 ** (-0.25 * rng.integers(0, 14, m))}[spread]   # on the bins' ends
    p = np.where(rng.random(m) < 0.5, p, 1.0 - p)
    codes = synth.apply_missing(rng, synth.hwe_genotypes(rng, p, n), 0.05)
    af = np.stack([p, 1.0 - p], 1)
    with kb.Estimator() as est:
        check(est, codes, oracle.relatedness(codes, af=af), af=af)


def test_chunks_leave_the_rows_unchanged(oracle):
    codes = cohort(140, 20_000, 9)
    with kb.Estimator() as est:
        whole = check(est, codes, oracle.relatedness(codes, num_samples=133), num_samples=133)
        est.set_launch(1000)       # chunks that end inside a sample's pairs
        parts = check(est, codes, whole, num_samples=133)
        assert est.run_stats()["slots"] == 1000
        est.set_launch(0)
        batch = est.relatedness_batch([(codes, None, 133), (cohort(20, 3000, 10), None, None), (codes, None, 7)])
    assert np.array_equal(whole.view(np.uint8), parts.view(np.uint8))
    assert np.array_equal(whole.view(np.uint8), batch[0].view(np.uint8))
    compare(batch[1], oracle.relatedness(cohort(20, 3000, 10)))


def test_pair_without_a_common_site(oracle):
    codes = cohort(5, 24_000, 11)
    codes[1, :12_000] = 3
    codes[3, 12_000:] = 3
    with kb.Estimator() as est:
        est.load(codes)
        rows = est.relatedness(allow_nosites=True)
        st = est.run_stats()
    assert st["fp64_passes"] == st["gh_passes"] > 0
    lone = (rows["x"] == 1) & (rows["y"] == 3)
    assert np.isnan(rows["obj"][lone]).all() and np.isnan(rows["jacquard"][lone]).all()
    assert np.isfinite(rows["obj"][~lone]).all()


@pytest.mark.parametrize("n,m", [(1, 200), (3, 129), (130, 4097)])
def test_cls_sizes(oracle, n, m):
    codes = synth.make_cohort(n, m, 800 + n, missing=0.0).codes
    ref = oracle.cls_relatedness(codes)
    with kb.Estimator() as est:
        est.load(codes)
        rows = est.relatedness_gt()
    compare(rows, ref)


def test_more_sites_of_a_frequency_than_a_32_bit_sum_holds():
    """17.3 million sites of one frequency and one genotype pair: the digit of -128
    that this frequency has in two of its columns adds up to -2.2e9.  The FP64 form
    (site lists) is the reference: the same sites, the objective at the shared bar
    (the overflow moved it by 1e-3, and its count of sites by 8e5)."""
    m, called = 17_600_000, 300_000
    codes = np.zeros((2, m), np.uint8)
    codes[:, :called] = np.random.default_rng(1).integers(0, 3, (2, called))
    af = np.empty((m, 2))
    af[:, 0] = 0.2622113028257064
    af[:, 1] = 1.0 - af[:, 0]
    got = {}
    for precision in ("fp32c", "fp64"):
        with kb.Estimator(precision=precision) as est:
            est.load(codes, af)
            got[precision] = est.relatedness(maf=0.0), est.run_stats()
    rows, st = got["fp32c"]
    ref, sr = got["fp64"]
    assert st["fp64_passes"] == st["gh_passes"] > 0 and st["pass_ms"] > 0, "the cohort should run on nodes"
    assert st["pair_sites"] == sr["pair_sites"] == 3 * m
    assert (np.abs(rows["obj"] - ref["obj"]) / np.abs(ref["obj"])).max() <= 1e-6


def test_split_bins_leave_the_rows_unchanged():
    """From 262,144 sites on, chunks of few pairs form a bin's weights in segments;
    the whole triangle (140 samples) does not: the sums are integers, so the rows
    are the same bit for bit."""
    codes = cohort(140, 270_000, 12)
    with kb.Estimator() as est:
        est.load(codes)
        whole = est.relatedness()
        assert est.run_stats()["fp64_passes"] == est.run_stats()["gh_passes"] > 0
        est.set_launch(1000)
        parts = est.relatedness()
        est.load(np.where(codes == 3, 0, codes))
        cls_parts = est.relatedness_gt()
        est.set_launch(0)
        cls_whole = est.relatedness_gt()
    assert np.array_equal(whole.view(np.uint8), parts.view(np.uint8))
    assert np.array_equal(cls_whole.view(np.uint8), cls_parts.view(np.uint8))


def test_calls_of_other_sizes_on_one_context():
    """One context keeps its slots, tables and graph while sizes grow and shrink (past
    4,096 pairs, past 16 and 64 cohorts in a call): the rows are a fresh context's."""
    sizes = [(5, 900), (130, 2100), (33, 4000), (2, 700), (95, 1000)]
    cohorts = {s: cohort(*s, 300 + s[0]) for s in sizes}
    small = [(cohort(3, 400, 900 + k), None, None) for k in range(70)]

    def calls(est, s):
        est.load(cohorts[s])
        complete = np.where(cohorts[s] == 3, 0, cohorts[s])
        ml = est.relatedness(allow_nosites=True)
        est.load(complete)
        return [ml, est.relatedness_gt(), est.relatedness(iterations=3, allow_nosites=True)]

    def batch(est, n):
        return est.relatedness_batch(small[:n])

    def fresh(f, arg):
        with kb.Estimator() as est:
            return f(est, arg)

    want = {s: fresh(calls, s) for s in sizes}
    want |= {n: fresh(batch, n) for n in (3, 20, 70)}
    with kb.Estimator() as est:
        for step in [*sizes, 3, *sizes[::-1], 20, sizes[3], 70, 3, sizes[1], 20, sizes[0]]:
            got = batch(est, step) if isinstance(step, int) else calls(est, step)
            for g, w in zip(got, want[step]):
                assert np.array_equal(g.view(np.uint8), w.view(np.uint8)), step


def test_frequencies_down_to_the_last_bin(oracle):
    """Frequencies from 2e-7 (the 64th bin) to 1/2, given by the caller, and one cohort
    just below, which stays on site lists."""
    n, m = 12, 9000
    rng = np.random.default_rng(15)
    p = np.exp(rng.uniform(np.log(2e-7), np.log(0.5), m))
    p[0] = 2e-7
    p = np.where(rng.random(m) < 0.5, p, 1.0 - p)
    codes = synth.apply_missing(rng, synth.hwe_genotypes(rng, p, n), 0.02)
    codes[:3, 0], codes[3, 0] = 0, 1     # the rarest allele is seen
    af = np.stack([p, 1.0 - p], 1)
    with kb.Estimator() as est:
        check(est, codes, oracle.relatedness(codes, af=af, maf=0.0), af=af, maf=0.0)
        af[0] = (1.8e-7, 1.0 - 1.8e-7)
        est.load(codes, af)
        est.relatedness(maf=0.0)
        assert est.run_stats()["fp64_passes"] < est.run_stats()["gh_passes"]


def test_rare_sites_at_the_default_cut(oracle):
    """300 samples, frequencies from the cut of 1/600 up, fitted on the device."""
    n, m = 300, 16_000
    rng = np.random.default_rng(16)
    p = np.exp(rng.uniform(np.log(1.0 / 600), np.log(0.5), m))
    p = np.where(rng.random(m) < 0.5, p, 1.0 - p)
    codes = synth.apply_missing(rng, synth.hwe_genotypes(rng, p, n), 0.05)
    with kb.Estimator() as est:
        check(est, codes, oracle.relatedness(codes, num_samples=50), num_samples=50)


def test_a_query_against_a_panel_in_chunks():
    """Chunks that end inside a query's row of pairs."""
    panel, query = cohort(150, 3000, 17), cohort(9, 3000, 18)
    rows = {}
    for slots in (0, 1000, 37):
        with kb.Estimator() as est:
            est.set_launch(slots)
            est.panel_load(panel)
            rows[slots] = est.wait(est.submit(query))
    assert np.array_equal(rows[0].view(np.uint8), rows[1000].view(np.uint8))
    assert np.array_equal(rows[0].view(np.uint8), rows[37].view(np.uint8))


def test_lists_where_the_node_layout_does_not_fit():
    """A cohort of few samples and many sites, with memory left for the lists' layout (57
    bytes a site, and 4 a listed site) but not for the nodes' (36 more): it is
    estimated on lists, as without them."""
    import torch
    n, m = 2, 40_000_000
    rng = np.random.default_rng(19)
    half = rng.integers(0, 3, (n, m // 8), dtype=np.uint8)
    codes = np.tile(half, (1, 8))
    small = cohort(n, 2000, 20)
    with kb.Estimator() as est:
        est.load(codes)
        want = est.relatedness(maf=0.0)
        assert est.run_stats()["fp64_passes"] == est.run_stats()["gh_passes"] > 0
    torch.cuda.empty_cache()
    with kb.Estimator() as est:
        est.load(small)
        est.relatedness(allow_nosites=True)
        est.set_precision("fp64")
        est.relatedness(allow_nosites=True)      # both engines' fixed parts are there
        est.set_precision("fp32c")
        free = torch.cuda.mem_get_info()[0]
        held = torch.empty(free - 57 * m - n * m - 18 * m, dtype=torch.uint8, device="cuda")
        est.load(codes)
        rows = est.relatedness(maf=0.0)
        assert est.run_stats()["fp64_passes"] < est.run_stats()["gh_passes"]
        del held
        torch.cuda.empty_cache()
    compare(rows, want)
