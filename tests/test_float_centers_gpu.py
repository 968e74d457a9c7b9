"""GPU parity of the float-center mode against the FP64 oracle.

The reference keeps uint8 centers (kmeans.cu:367); this mode keeps fp32 centers computed in FP64
from exact integer sums, takes distances from the tensor cores with fixed-point centers (hi + lo bf16
parts outside [0, 256)) or, for few descriptors, from fp32 differences, and re-scores in FP64 every
descriptor whose margin is within the error bound of its form.  So
the assignments -- and therefore the centers, occurrence counts and word IDs -- must be identical
to the oracle's FP64 evaluation (oracle/rbw_oracle.cpp, orc_build_vocabulary_f32 /
orc_lookup_f32), and centers within 1e-5 relative of its FP64 means."""
import os

import numpy as np
import pytest
import torch

import rapidbow_b200 as rbw
from oracle.pyoracle import INIT_INJECTED, INIT_KMEANSPP, level_beg
from rapidbow_b200.synth import sift_like
from tests.helpers import edge_descriptors, random_tree

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


def _lookup(voc, desc_np):
    out = voc.lookup(torch.from_numpy(desc_np).cuda())
    torch.cuda.synchronize()
    assert voc.device_errors() == (0, 0)
    return out.cpu().numpy().view(np.uint32)


def _rel(a, b):
    a = a.astype(np.float64)
    b = b.astype(np.float64)
    return float(np.max(np.abs(a - b) / np.maximum(np.abs(b), 1e-30)))


def test_integer_valued_float_tree_equals_uint8_tree(oracle):
    """fp32 centers holding integers: FP64 distances are exact integers, so the float lookup must
    equal the uint8 lookup of the same tree, duplicate centers (exact ties) included."""
    for B, L, seed in [(16, 3, 1), (10, 4, 2), (3, 6, 3)]:
        centers, masks, weights = random_tree(B, L, seed=seed, dup_rate=0.3)
        v8 = rbw.vocabulary_from_host(B, L, centers, masks, weights)
        vf = rbw.vocabulary_from_host_f32(B, L, centers.astype(np.float32), masks, weights)
        assert vf.float_centers and not v8.float_centers
        desc = edge_descriptors(centers, 20011, seed=seed + 10)
        want = oracle.lookup(centers, B, L, desc, threads=THREADS)
        assert np.array_equal(_lookup(v8, desc), want)
        assert np.array_equal(_lookup(vf, desc), want)
        assert np.array_equal(oracle.lookup_f32(centers.astype(np.float32), B, L, desc, threads=THREADS), want)
        assert vf.refined_lookups() > 0  # exact ties are always re-scored


def test_float_lookup_near_ties_match_fp64_oracle(oracle):
    """Pairs of centers that differ by a fraction of a unit in a few dimensions put many
    descriptors within the error bound; the re-score must settle each of them exactly as FP64."""
    rng = np.random.default_rng(5)
    data = sift_like(40000, seed=5).numpy()
    B, L = 16, 3
    nodes = level_beg(B, L)
    centers = data[rng.integers(0, data.shape[0], nodes * B)].reshape(nodes, B, 128).astype(np.float32)
    centers += rng.uniform(-0.5, 0.5, centers.shape).astype(np.float32)
    for b in range(1, B, 2):  # odd centers: near copies of the even ones
        centers[:, b] = centers[:, b - 1]
        centers[:, b, :4] += rng.uniform(-0.05, 0.05, (nodes, 4)).astype(np.float32)
    masks = np.full(nodes, (1 << B) - 1, np.uint32)
    weights = np.ones((nodes, B), np.float32)
    voc = rbw.vocabulary_from_host_f32(B, L, centers, masks, weights)
    desc = np.concatenate([data, sift_like(60000, seed=6).numpy()])
    voc.refined_lookups()
    got = _lookup(voc, desc)
    refined = voc.refined_lookups()
    want = oracle.lookup_f32(centers, B, L, desc, threads=THREADS)
    assert np.array_equal(got, want), f"{np.count_nonzero(got != want)} of {got.size} differ"
    # every center has a near copy, so nearly every descriptor is re-scored at every level
    assert 0.5 * 3 * desc.shape[0] < refined <= 3 * desc.shape[0]


def test_float_blob_round_trip_and_rounded_tree():
    rng = np.random.default_rng(7)
    B, L = 10, 3
    nodes = level_beg(B, L)
    centers = rng.uniform(0, 255, (nodes, B, 128)).astype(np.float32)
    masks = np.full(nodes, (1 << B) - 1, np.uint32)
    weights = rng.uniform(0.1, 2, (nodes, B)).astype(np.float32)
    voc = rbw.vocabulary_from_host_f32(B, L, centers, masks, weights)
    blob = voc.serialize()
    voc2 = rbw.deserialize_vocabulary(blob)
    assert voc2.float_centers
    assert np.array_equal(voc2.centers_f32(), centers)
    assert voc2.serialize() == blob
    c8, m, w = voc2.tree()
    assert np.array_equal(c8, np.clip(np.rint(centers), 0, 255).astype(np.uint8))
    assert np.array_equal(m, masks) and np.array_equal(w, weights)
    with pytest.raises(rbw.RbwError) as e:
        rbw.deserialize_vocabulary(blob[:-4])
    assert e.value.status == rbw.RBW_ERR_INVALID_BLOB
    with pytest.raises(rbw.RbwError) as e:
        voc.lookup_noalloc(torch.zeros((4, 128), dtype=torch.uint8, device="cuda"),
                           torch.zeros(4, dtype=torch.int32, device="cuda"))
    assert e.value.status == rbw.RBW_ERR_UNSUPPORTED
    with pytest.raises(rbw.RbwError) as e:
        rbw.vocabulary_from_host(B, L, c8, masks, weights).centers_f32()
    assert e.value.status == rbw.RBW_ERR_UNSUPPORTED


def _check_float_build(oracle, desc, B, L, init, seed=0, injected=None, fresh=None):
    dev = torch.from_numpy(desc).cuda()
    voc = rbw.build_vocabulary(dev, B, nb_doc=1000, nb_levels=L, init=init, seed=seed, injected=injected,
                               max_iterations=10, check_interval=4, float_centers=True)
    ref = oracle.build_vocabulary_f32(desc, 1000, B, L, max_iter=10,
                                      init={"kmeans++": INIT_KMEANSPP, "injected": INIT_INJECTED}[init], seed=seed,
                                      injected=injected, threads=THREADS)
    got = voc.centers_f32()
    assert _rel(got, ref["centers"]) <= 1e-5
    assert np.array_equal(got, ref["centers"]), "centers differ from the FP64 oracle"
    c8, masks, weights = voc.tree()
    assert np.array_equal(masks, ref["masks"])
    assert np.array_equal(weights, ref["weights"]), "occurrence counts (assignments) differ"
    st = voc.build_stats()
    assert st["levels"] == L
    for lv in range(L):
        assert abs(st["inertia_first"][lv] - ref["inertia_first"][lv]) <= 1e-9 * ref["inertia_first"][lv]
        assert abs(st["inertia_last"][lv] - ref["inertia_last"][lv]) <= 1e-9 * ref["inertia_last"][lv]
        assert st["inertia_last"][lv] <= st["inertia_first"][lv]
        assert st["refined"][lv] <= st["assignments"][lv]
    assert sum(st["refined"]) > 0
    for x in [desc] + ([fresh] if fresh is not None else []):
        assert np.array_equal(_lookup(voc, x), oracle.lookup_f32(ref["centers"], B, L, x, threads=THREADS))
    return voc, ref, st


def test_float_build_matches_fp64_oracle_b16(oracle):
    desc = sift_like(60000, seed=31).numpy()
    _check_float_build(oracle, desc, 16, 3, "kmeans++", seed=9, fresh=sift_like(20000, seed=32).numpy())


def test_float_build_zipf_1m_b10_l4_injected_init(oracle):
    """The 10M-descriptor, 4,096-component Zipf(1.1) workload's generator at 1M descriptors, a
    10-ary, 4-level tree, injected initial centers (random descriptor rows, some slots invalid)
    and 10 Lloyd iterations."""
    B, L = 10, 4
    n = 1_000_000
    desc = sift_like(n, seed=41, n_components=4096, zipf=1.1, device="cuda").cpu().numpy()
    rng = np.random.default_rng(42)
    nodes = level_beg(B, L)
    injected = rng.integers(0, n, (nodes, B)).astype(np.uint32)
    injected[rng.random(nodes) < 0.05, B - 1] = 0xFFFFFFFF  # an invalid last slot in 5% of the nodes
    fresh = sift_like(200_000, seed=43, n_components=4096, zipf=1.1, device="cuda").cpu().numpy()
    _check_float_build(oracle, desc, B, L, "injected", injected=injected, fresh=fresh)


def test_uint8_build_injected_init_matches_oracle(oracle):
    """The uint8 mode with injected initial centers (RBW_INIT_INJECTED) on the Zipf generator:
    byte-identical to the oracle (IEEE rounding of the quotient, as the oracle divides)."""
    B, L = 10, 4
    n = 300_000
    desc = sift_like(n, seed=51, n_components=4096, zipf=1.1, device="cuda").cpu().numpy()
    rng = np.random.default_rng(52)
    nodes = level_beg(B, L)
    injected = rng.integers(0, n, (nodes, B)).astype(np.uint32)
    injected[rng.random(nodes) < 0.05, B - 1] = 0xFFFFFFFF
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=1000, nb_levels=L, init="injected",
                               injected=injected, max_iterations=10, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 1000, B, L, max_iter=10, init=INIT_INJECTED, injected=injected)
    c, m, w = voc.tree()
    assert np.array_equal(c, ref["centers"])
    assert np.array_equal(m, ref["masks"])
    assert np.array_equal(w, ref["weights"])
    assert np.array_equal(_lookup(voc, desc), oracle.lookup(ref["centers"], B, L, desc, threads=THREADS))


@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (255.99 / 255, 0.0), (3.0, -100.0), (1.0, -0.001), (1.01, 0.0)])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 48_000, 48_001])
def test_float_lookup_inside_and_outside_the_fixed_point_range(oracle, scale, shift, n):
    """Centers in [0, 256) take the fixed-point operand, any other value the bf16 one; both equal FP64,
    near ties (copies of rows among the centers) included."""
    rng = np.random.default_rng(n)
    B, L = 10, 3
    nodes = level_beg(B, L)
    data = sift_like(3000, seed=61).numpy()
    centers = data[rng.integers(0, data.shape[0], nodes * B)].reshape(nodes, B, 128).astype(np.float32)
    centers[:, 1::2] += rng.uniform(0, 0.02, centers[:, 1::2].shape).astype(np.float32)
    centers[0, 0, 0] = 255.0
    centers = (centers * np.float32(scale) + np.float32(shift)).astype(np.float32)
    voc = rbw.vocabulary_from_host_f32(B, L, centers, np.full(nodes, 1023, np.uint32), np.ones((nodes, B), np.float32))
    desc = np.concatenate([data, edge_descriptors(np.clip(centers, 0, 255).astype(np.uint8), 48_001, 62)])[-n:]
    assert np.array_equal(_lookup(voc, np.ascontiguousarray(desc)), oracle.lookup_f32(centers, B, L, desc, threads=THREADS))


@pytest.mark.parametrize("n_distinct,n", [(3, 700), (40, 30_000), (500, 9_000)])
def test_float_build_of_duplicated_rows_matches_fp64_oracle(oracle, n_distinct, n):
    """Few distinct rows: exact ties in most tiles, so the queue of members to settle in FP64 fills
    within a node and at its end, in one node over many CTAs and in small ones."""
    base = sift_like(n_distinct, seed=71 + n_distinct).numpy()
    base[1] = base[0]
    base[1, :2] += 1
    desc = np.ascontiguousarray(base[np.random.default_rng(n).integers(0, n_distinct, n)])
    B, L = 10, 2
    rng = np.random.default_rng(n + 1)
    injected = rng.integers(0, n, (level_beg(B, L), B)).astype(np.uint32)
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=30, nb_levels=L, init="injected",
                               injected=injected, max_iterations=5, check_interval=2, float_centers=True)
    ref = oracle.build_vocabulary_f32(desc, 30, B, L, max_iter=5, init=INIT_INJECTED, injected=injected, threads=THREADS)
    assert np.array_equal(voc.centers_f32(), ref["centers"])
    assert np.array_equal(voc.tree()[2], ref["weights"])
    st = voc.build_stats()
    for lv in range(L):
        assert abs(st["inertia_last"][lv] - ref["inertia_last"][lv]) <= 1e-9 * max(ref["inertia_last"][lv], 1.0)


@pytest.mark.parametrize("B,L,n", [(16, 1, 16_001), (2, 8, 140_003), (16, 5, 90_001), (10, 4, 64_001), (3, 3, 250_000)])
def test_float_lookup_by_levels_matches_fp64_oracle(oracle, B, L, n):
    """Above the one-launch limit: children counted by the assign and scanned in one CTA, or (trees
    with more than 32,768 last-level nodes) regrouped as builds do; empty nodes in most levels."""
    centers, masks, weights = random_tree(B, L, seed=B + L, dup_rate=0.2)
    centers = centers.astype(np.float32)
    centers[:, 1::2] = np.minimum(centers[:, 1::2] + np.float32(0.25), 255)
    voc = rbw.vocabulary_from_host_f32(B, L, centers, masks, weights)
    desc = edge_descriptors(centers.astype(np.uint8), n, seed=n)
    assert np.array_equal(_lookup(voc, desc), oracle.lookup_f32(centers, B, L, desc, threads=THREADS))


@pytest.mark.parametrize("scale", [1e-20, 0.001, 0.003, 0.03, 0.3])
@pytest.mark.parametrize("bright", [False, True])
def test_float_lookup_of_centers_much_shorter_than_the_rows(oracle, scale, bright):
    """Centers in [0, scale) and rows of |x| near 500 or near 2,300 (a few of them zero): distances that
    agree in their leading bits.  The words are FP64's in the one-launch descent and level by level, on
    both sides of the limit between them (16,000 rows per level)."""
    rng = np.random.default_rng(int(bright))
    B, n = 10, 16_001
    centers = (rng.random((1, B, 128)) * scale).astype(np.float32)
    desc = rng.integers(150, 256, (n, 128), dtype=np.uint8) if bright else sift_like(n, seed=63).numpy()
    desc[:3] = 0
    voc = rbw.vocabulary_from_host_f32(B, 1, centers, np.full(1, 1023, np.uint32), np.ones((1, B), np.float32))
    want = oracle.lookup_f32(centers, B, 1, desc, threads=THREADS)
    for m in (700, n - 1, n):
        got = _lookup(voc, desc[:m])
        assert voc.last_kernels == 1 if m < n else voc.last_kernels > 1
        assert np.array_equal(got, want[:m]), f"{m} rows: {np.count_nonzero(got != want[:m])} differ"


@pytest.mark.parametrize("n", [700, 40_001])
def test_centers_that_are_no_numbers_are_never_nearest(oracle, n):
    """NaN centers in any slot but the first, among near ties that FP64 settles: every word is that of
    the nearest of the others, as in the oracle."""
    rng = np.random.default_rng(n)
    B, L = 10, 3
    nodes = level_beg(B, L)
    data = sift_like(3000, seed=65).numpy()
    centers = data[rng.integers(0, data.shape[0], nodes * B)].reshape(nodes, B, 128).astype(np.float32)
    centers[:, 1::2] = centers[:, 0::2] + rng.uniform(0, 0.01, centers[:, 0::2].shape).astype(np.float32)
    lost = rng.random((nodes, B)) < 0.25
    lost[:, 0] = False
    centers[lost] = np.nan
    voc = rbw.vocabulary_from_host_f32(B, L, centers, np.full(nodes, 1023, np.uint32), np.ones((nodes, B), np.float32))
    desc = np.ascontiguousarray(data[rng.integers(0, data.shape[0], n)])
    voc.refined_lookups()
    assert np.array_equal(_lookup(voc, desc), oracle.lookup_f32(centers, B, L, desc, threads=THREADS))
    assert voc.refined_lookups() > 0
