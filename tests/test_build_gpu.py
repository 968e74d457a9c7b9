"""GPU hierarchical k-means build (Vocabulary.cpp:32-121, kmeans.cpp) against the oracle and the
reference's own build.

The reference rounds centers with its --use_fast_math division (kmeans.cu:367); the oracle
divides with IEEE division.  Comparisons with the oracle therefore build with
ieee_division=True, and the default (reference) rounding is pinned against the reference's own
build, bit for bit."""
import numpy as np
import pytest
import torch

import rapidbow_b200 as rbw
from oracle.pyoracle import INIT_KMEANSPP, INIT_REFERENCE, parse_reference_blob
from rapidbow_b200.synth import sift_like

pytestmark = pytest.mark.gpu


def _tree_equal(voc, ref):
    c, m, w = voc.tree()
    assert np.array_equal(m, ref["masks"]), "masks differ"
    bad = np.argwhere(c != ref["centers"])
    assert bad.size == 0, f"{len(bad)} center bytes differ, first at {bad[:3].tolist()}"
    assert np.array_equal(w, ref["weights"]), "weights differ"


@pytest.mark.parametrize("B,L,n", [(16, 2, 3000), (16, 3, 20000), (10, 3, 8000), (4, 4, 1500)])
def test_build_reference_init_matches_oracle(oracle, B, L, n):
    desc = sift_like(n, seed=B + L).numpy()
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=77, nb_levels=L, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 77, B, L, max_iter=1000, init=INIT_REFERENCE)
    _tree_equal(voc, ref)


@pytest.mark.parametrize("B,L,n,iters", [(16, 3, 20000, 10), (10, 3, 10000, 10), (16, 2, 5000, 1000)])
def test_build_kmeanspp_matches_oracle(oracle, B, L, n, iters):
    desc = sift_like(n, seed=100 + B).numpy()
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=50, nb_levels=L, init="kmeans++", seed=1234,
                               max_iterations=iters, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 50, B, L, max_iter=iters, init=INIT_KMEANSPP, seed=1234)
    _tree_equal(voc, ref)


@pytest.mark.parametrize("n_distinct,n", [(6, 3000), (40, 600), (300, 5000)])
def test_build_kmeanspp_duplicates_match_oracle(oracle, n_distinct, n):
    """Few distinct rows: the D^2 weights reach zero before B picks (fewer valid centers, empty
    children at the next level) and the sampled candidates repeat."""
    base = sift_like(n_distinct, seed=321 + n_distinct).numpy()
    desc = np.ascontiguousarray(base[np.random.default_rng(n).integers(0, n_distinct, n)])
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), 16, nb_doc=20, nb_levels=2, init="kmeans++", seed=99,
                               max_iterations=10, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 20, 16, 2, max_iter=10, init=INIT_KMEANSPP, seed=99)
    _tree_equal(voc, ref)


def test_build_matches_reference_build(reference):
    """Bit-identical blob with the reference's own buildVocabulary (same default-seeded RNG)."""
    desc = sift_like(30000, seed=77).numpy()
    blob_ref = reference.build_vocabulary(desc, nb_doc=123, L=3)
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), 16, nb_doc=123, nb_levels=3)
    blob = voc.serialize()
    if blob != blob_ref:
        L, c, m, w = parse_reference_blob(blob_ref)
        _tree_equal(voc, dict(centers=c, masks=m, weights=w))
    assert blob == blob_ref


def test_build_matches_reference_build_ten_iterations(reference):
    desc = sift_like(20000, seed=78).numpy()
    blob_ref = reference.build_vocabulary(desc, nb_doc=10, L=3, max_iter=10, check_interval=4)
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), 16, nb_doc=10, nb_levels=3, max_iterations=10)
    assert voc.serialize() == blob_ref


def test_ref_check_full_every_descriptor_is_its_own_leaf():
    """tests/VocTests.cpp:86-132: 32 random descriptors, 3 levels -> inertia 0."""
    rng = np.random.default_rng(0)
    desc = rng.integers(0, 256, size=(32, 128), dtype=np.uint8)
    d = torch.from_numpy(desc).cuda()
    voc = rbw.build_vocabulary(d, 16, nb_doc=4, nb_levels=3)
    leaf = voc.lookup(d).cpu().numpy().view(np.uint32)
    c, _, _ = voc.tree()
    leaves = c[1 + 16:].reshape(-1, 128)
    assert np.all(leaves[leaf] == desc)


def test_ref_check_2d_rms_below_ten():
    """tests/VocTests.cpp:38-84: only bytes 126-127 random, 2 levels -> RMS to leaf <= 10."""
    rng = np.random.default_rng(0)
    desc = np.zeros((4096, 128), np.uint8)
    desc[:, 126:128] = rng.integers(0, 256, size=(4096, 2), dtype=np.uint8)
    d = torch.from_numpy(desc).cuda()
    voc = rbw.build_vocabulary(d, 16, nb_doc=16, nb_levels=2)
    leaf = voc.lookup(d).cpu().numpy().view(np.uint32)
    c, _, _ = voc.tree()
    cent = c[1:].reshape(-1, 128)[leaf].astype(np.int64)
    rms = np.sqrt(((desc.astype(np.int64) - cent) ** 2).sum(1).mean())
    assert rms <= 10


def test_build_rejects_bad_input():
    d = torch.zeros((10, 128), dtype=torch.uint8, device="cuda")
    with pytest.raises(rbw.RbwError) as e:
        rbw.build_vocabulary(d, 16, nb_doc=1, nb_levels=2)
    assert "Insufficient descriptors" in str(e.value)
    d = torch.zeros((100, 128), dtype=torch.uint8, device="cuda")
    with pytest.raises(rbw.RbwError):
        rbw.build_vocabulary(d, 16, nb_doc=0, nb_levels=2)
    with pytest.raises(rbw.RbwError) as e:
        rbw.build_vocabulary(d, 17, nb_doc=1, nb_levels=2)
    assert e.value.status == rbw.RBW_ERR_UNSUPPORTED


@pytest.mark.parametrize("B,n", [(2, 127), (3, 128), (16, 129), (10, 255), (16, 257), (7, 94_721), (16, 189_440 + 33)])
def test_build_tile_edges_match_oracle(oracle, B, n):
    """Nodes of one tile, one row more or less, and one node over every CTA (one and two tiles per
    CTA of five on each SM, ragged): assignment, change counts and center sums of the two MMAs."""
    desc = sift_like(n, seed=n).numpy()
    for level_members in (desc, np.repeat(desc[: max(B, n // 50)], 7, axis=0)):  # distinct, duplicated rows
        voc = rbw.build_vocabulary(torch.from_numpy(np.ascontiguousarray(level_members)).cuda(), B, nb_doc=50,
                                   nb_levels=2, init="kmeans++", seed=4, max_iterations=6, ieee_division=True)
        ref = oracle.build_vocabulary(level_members, 50, B, 2, max_iter=6, init=INIT_KMEANSPP, seed=4)
        _tree_equal(voc, ref)


@pytest.mark.parametrize("n", [16, 128, 129, 256, 257, 767, 768, 769, 1535, 1536, 1537])
@pytest.mark.parametrize("B,iters,check", [(16, 1000, 4), (5, 7, 3)])
def test_build_resident_node_sizes_match_oracle(oracle, n, B, iters, check):
    """Nodes at the edges of the classes whose whole Lloyd loop runs in one CTA, and one row above
    the largest (streamed); the level's step count is the one of a loop polled every `check` steps."""
    desc = sift_like(n, seed=n + B).numpy()
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=30, nb_levels=2, max_iterations=iters,
                               check_interval=check, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 30, B, 2, max_iter=iters, init=INIT_REFERENCE)
    _tree_equal(voc, ref)
    stops = [ref["iters"][:1].max(), ref["iters"][1:].max()]  # the step that changed nothing, per level
    want = [min(iters, -(-int(s) // check) * check) for s in stops]
    assert voc.build_stats()["iterations"] == want


@pytest.mark.parametrize("B,L,n", [(16, 4, 20_011), (8, 5, 9_000), (9, 5, 9_000), (2, 8, 70_001), (16, 2, 33)])
def test_build_tile_lists_and_children_match_oracle(oracle, B, L, n):
    """Levels of up to 4,096 nodes, whose tile list is one launch, and of more; many nodes without
    members."""
    desc = sift_like(n, seed=n + B).numpy()
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=40, nb_levels=L, init="kmeans++", seed=5,
                               max_iterations=4, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 40, B, L, max_iter=4, init=INIT_KMEANSPP, seed=5)
    _tree_equal(voc, ref)


@pytest.mark.parametrize("B,L,n,distinct", [(4, 6, 60_000, 0), (11, 4, 100_003, 0), (16, 4, 200_001, 900)])
def test_build_kmeanspp_small_nodes_match_oracle(oracle, B, L, n, distinct):
    """Levels of 1,000 and more small nodes, where a warp seeds a node of at most 128 members and a CTA
    each larger one; repeated rows (weights that reach zero)."""
    desc = sift_like(distinct or n, seed=n + B).numpy()
    if distinct:
        desc = np.ascontiguousarray(desc[np.random.default_rng(n).integers(0, distinct, n) ** 2 % distinct])
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=40, nb_levels=L, init="kmeans++", seed=6,
                               max_iterations=3, ieee_division=True)
    ref = oracle.build_vocabulary(desc, 40, B, L, max_iter=3, init=INIT_KMEANSPP, seed=6)
    _tree_equal(voc, ref)


@pytest.mark.parametrize("rows_per_sm,extra,L", [(12, -1, 2), (1536, 0, 1), (1536, 1, 1), (400, 77, 2)])
def test_build_shared_level_edges_match_oracle(oracle, rows_per_sm, extra, L):
    """Levels whose streamed rows fit the SMs together run in one cooperative launch, nodes spread
    over the CTAs (up to 1,536 rows per SM); one row more is streamed step by step."""
    n = torch.cuda.get_device_properties(0).multi_processor_count * rows_per_sm + extra
    desc = sift_like(n, seed=rows_per_sm).numpy()
    B = 6
    voc = rbw.build_vocabulary(torch.from_numpy(desc).cuda(), B, nb_doc=30, nb_levels=L, max_iterations=9,
                               ieee_division=True)
    ref = oracle.build_vocabulary(desc, 30, B, L, max_iter=9, init=INIT_REFERENCE)
    _tree_equal(voc, ref)
    assert voc.build_stats()["iterations"][0] == min(9, -(-int(ref["iters"][0]) // 4) * 4)


@pytest.mark.parametrize("n,L", [(1_000, 2), (20_000, 2), (150_000, 3)])
def test_build_in_a_context_of_some_of_the_sms_matches_oracle(oracle, n, L):
    """A stream whose context owns part of the SMs cannot run one cooperative launch over all of them:
    levels whose nodes would be spread over the CTAs are streamed, small nodes run in their classes."""
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]

    torch.zeros(1, device="cuda")
    dev = ok(driver.cuDeviceGet(torch.cuda.current_device()))
    sms = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    part = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, sms.sm.smCount // 2))[0][0]
    context = ok(driver.cuGreenCtxCreate(ok(driver.cuDevResourceGenerateDesc([part], 1)), dev,
                                         driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(context, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    desc = sift_like(n, seed=n).numpy()
    rows = torch.from_numpy(desc).cuda()
    torch.cuda.synchronize()
    B = 8
    voc = rbw.build_vocabulary(rows, B, nb_doc=30, nb_levels=L, max_iterations=9, ieee_division=True, stream=int(stream))
    ref = oracle.build_vocabulary(desc, 30, B, L, max_iter=9, init=INIT_REFERENCE)
    _tree_equal(voc, ref)
    beg = [sum(B ** i for i in range(level)) for level in range(L + 1)]
    assert voc.build_stats()["iterations"] == [min(9, -(-int(max(ref["iters"][a:b])) // 4) * 4)
                                               for a, b in zip(beg, beg[1:])]
    del voc
    ok((driver.cuStreamDestroy(stream)[0], None))
    ok((driver.cuGreenCtxDestroy(context)[0], None))
    other = rbw.build_vocabulary(rows, B, nb_doc=30, nb_levels=L, max_iterations=9, ieee_division=True)
    _tree_equal(other, ref)  # no error is left behind


def test_a_refused_build_leaves_no_error_behind():
    """A tree too large for any GPU (15^8 words) is refused with RBW_ERR_OUT_OF_MEMORY; the calls after
    it work."""
    desc = sift_like(2_000, seed=1, device="cuda")
    voc = rbw.build_vocabulary(desc, 10, nb_doc=10, nb_levels=2, init="kmeans++", max_iterations=3)
    want, words = voc.tree()[0], voc.lookup(desc).clone()
    calls = [lambda: np.array_equal(voc.tree()[0], want), lambda: torch.equal(voc.lookup(desc), words),
             lambda: rbw.build_vocabulary(desc, 10, nb_doc=10, nb_levels=1).nb_levels == 1]
    for call in calls:
        with pytest.raises(rbw.RbwError) as e:
            rbw.build_vocabulary(desc, 15, nb_doc=10, nb_levels=8)
        assert e.value.status == rbw.RBW_ERR_OUT_OF_MEMORY
        assert call()
