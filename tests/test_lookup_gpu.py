"""GPU parity of the tree descent (vocTreeLookUp.cu:82-155 semantics): word IDs must be
bit-identical to the oracle and to the reference's own kernel, for every algorithm."""
import numpy as np
import pytest
import torch

import rapidbow_b200 as rbw
from tests.helpers import edge_descriptors, random_tree

pytestmark = pytest.mark.gpu

ALGOS = ["tensor_u8", "simt_f32", "tensor_u8_warpnode", "tensor_u8_ring"]


def _lookup(voc, desc_np, algo):
    d = torch.from_numpy(desc_np).cuda()
    out = voc.lookup(d, algo=algo)
    torch.cuda.synchronize()
    assert voc.device_errors() == (0, 0)
    return out.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("B,L", [(16, 1), (16, 2), (16, 3), (16, 4), (10, 3), (10, 4), (2, 7), (3, 5), (16, 5)])
@pytest.mark.parametrize("algo", ALGOS)
def test_lookup_matches_oracle(oracle, B, L, algo):
    centers, masks, weights = random_tree(B, L, seed=B * 100 + L)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    for n, seed in [(1, 1), (17, 2), (129, 3), (4099, 4)]:
        desc = edge_descriptors(centers, n, seed)
        got = _lookup(voc, desc, algo)
        want = oracle.lookup(centers, B, L, desc)
        assert np.array_equal(got, want), f"n={n}: {np.count_nonzero(got != want)} mismatches"


@pytest.mark.parametrize("n", [0, 1, 15, 16, 127, 128, 129, 255, 256, 257, 100003, 2000003])
def test_lookup_sizes_tensor_vs_simt_vs_oracle(oracle, n):
    B, L = 16, 4
    centers, masks, weights = random_tree(B, L, seed=7)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = edge_descriptors(centers, n, seed=n)
    a = _lookup(voc, desc, "tensor_u8")
    b = _lookup(voc, desc, "simt_f32")
    assert np.array_equal(a, b)
    assert np.array_equal(_lookup(voc, desc, "tensor_u8_warpnode"), b)
    assert np.array_equal(_lookup(voc, desc, "tensor_u8_ring"), b)
    assert np.array_equal(a, oracle.lookup(centers, B, L, desc, threads=8))


def test_lookup_ties_all_equal_descriptors_and_extremes(oracle):
    B, L = 16, 3
    centers, masks, weights = random_tree(B, L, seed=11, dup_rate=0.5)
    centers[0, :] = centers[0, 5]          # root: every center identical -> branch 0 always
    centers[1, 3] = 0
    centers[1, 4] = 255
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = np.concatenate([np.zeros((300, 128), np.uint8), np.full((300, 128), 255, np.uint8),
                           np.tile(centers[1, 7], (300, 1))])
    for algo in ALGOS:
        got = _lookup(voc, desc, algo)
        assert np.array_equal(got, oracle.lookup(centers, B, L, desc))
        assert np.all(got // 256 == 0)  # tie at the root resolves to branch 0


def test_lookup_sift_like_tree(oracle):
    from rapidbow_b200.synth import sift_like

    data = sift_like(20000, seed=5).numpy()
    B, L = 16, 4
    centers, masks, weights = random_tree(B, L, seed=3, data=data)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = sift_like(50000, seed=6).numpy()
    want = oracle.lookup(centers, B, L, desc, threads=8)
    for algo in ALGOS:
        assert np.array_equal(_lookup(voc, desc, algo), want)


def test_lookup_matches_reference_kernel(reference):
    """The reference's own kernel (built for sm_100a in oracle/_ref) on the same blob."""
    from rapidbow_b200.synth import sift_like

    data = sift_like(20000, seed=8).numpy()
    B, L = 16, 4
    centers, masks, weights = random_tree(B, L, seed=9, data=data)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    blob = voc.serialize()
    desc = np.concatenate([sift_like(30000, seed=10).numpy(), edge_descriptors(centers, 3000, 12)])
    want = reference.lookup(blob, desc)
    for algo in ALGOS:
        assert np.array_equal(_lookup(voc, desc, algo), want)


def test_lookup_host_pipeline_matches_device_path(oracle):
    B, L = 16, 4
    centers, masks, weights = random_tree(B, L, seed=21)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = edge_descriptors(centers, (1 << 20) + 12345, seed=22)
    got = voc.lookup_host(desc)
    assert np.array_equal(got, oracle.lookup(centers, B, L, desc, threads=8))


def test_blob_round_trip_is_byte_exact():
    B, L = 16, 3
    centers, masks, weights = random_tree(B, L, seed=31)
    masks[5] = 0x00FF
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    blob = voc.serialize()
    assert len(blob) == 4 + (1 + 16 + 256) * (2048 + 2 + 64)
    voc2 = rbw.deserialize_vocabulary(blob)
    assert voc2.serialize() == blob
    c, m, w = voc2.tree()
    assert np.array_equal(c, centers) and np.array_equal(m, masks) and np.array_equal(w, weights)
    with pytest.raises(rbw.RbwError) as e:
        rbw.deserialize_vocabulary(blob[:-1])
    assert e.value.status == rbw.RBW_ERR_INVALID_BLOB


def test_blob_extension_for_other_branch_factors():
    B, L = 10, 3
    centers, masks, weights = random_tree(B, L, seed=41)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    voc2 = rbw.deserialize_vocabulary(voc.serialize())
    assert voc2.branch_factor == 10 and voc2.nb_levels == 3
    c, m, w = voc2.tree()
    assert np.array_equal(c, centers) and np.array_equal(w, weights)


def test_lookup_repeated_large_batches_are_exact():
    """Many centre groups per CTA in the gathered pass and a producer that runs ahead of the
    MMA: the double-buffered centre blocks and the row-index ring are reused as fast as the
    hardware allows.  Every repetition must equal the FP32 kernel exactly."""
    from rapidbow_b200.synth import sift_like

    train = sift_like(500_000, seed=21, device="cuda")
    voc = rbw.build_vocabulary(train, 16, nb_doc=1000, nb_levels=4, init="kmeans++", seed=5, max_iterations=5)
    desc = sift_like(8_000_000, seed=22, device="cuda")
    want = voc.lookup(desc, algo="simt_f32")
    for algo in ("tensor_u8", "tensor_u8_warpnode", "tensor_u8_ring"):
        for _ in range(4):
            got = voc.lookup(desc, algo=algo)
            torch.cuda.synchronize()
            assert voc.device_errors() == (0, 0)
            assert int((got != want).sum()) == 0, algo


@pytest.mark.parametrize("B,L", [(2, 8), (3, 2), (5, 4), (9, 3), (10, 6), (12, 1), (13, 4), (16, 3), (16, 4)])
def test_auto_lookup_matches_oracle_on_both_sides_of_the_direct_limit(oracle, B, L):
    """Few rows go down the tree in one launch (a warp per row, ragged last block), more through
    the tensor-core passes: the same words, ties included, and as many launches as that path has."""
    centers, masks, weights = random_tree(B, L, seed=B + L, dup_rate=0.3)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    limit = 32768 if L <= 2 else 100000 if L <= 4 else 200000
    for n in (1, 2, 3, 4, 5, 31, 733, limit, limit + 1):
        desc = edge_descriptors(centers, n, seed=n)
        got = _lookup(voc, desc, "auto")
        assert (voc.last_kernels == 1) == (n <= limit or L <= 2)
        want = oracle.lookup(centers, B, L, desc, threads=8)
        assert np.array_equal(got, want), f"n={n}: {np.count_nonzero(got != want)} mismatches"


@pytest.mark.parametrize("B,limit", [(2, 150_000), (4, 150_000), (5, 200_000)])
def test_auto_lookup_limit_of_six_levels(oracle, B, limit):
    """Six levels whose regroups are all small (B <= 4) go to the tensor cores from fewer rows on."""
    centers, masks, weights = random_tree(B, 6, seed=B, dup_rate=0.3)
    voc = rbw.vocabulary_from_host(B, 6, centers, masks, weights)
    for n in (limit, limit + 1):
        desc = edge_descriptors(centers, n, seed=n)
        got = _lookup(voc, desc, "auto")
        assert (voc.last_kernels == 1) == (n == limit)
        assert np.array_equal(got, oracle.lookup(centers, B, 6, desc, threads=8))


@pytest.mark.parametrize("B,L", [(2, 4), (5, 3), (13, 2), (14, 2), (16, 1), (16, 2), (16, 3), (16, 4)])
def test_sorted_passes_match_oracle(oracle, B, L):
    """Tensor-core passes around the 128-row tiles and 256-row super-tiles, with all rows on one branch
    and with rows on every branch, with children areas for both teams (B <= 13) and one shared."""
    centers, masks, weights = random_tree(B, L, seed=B * L, dup_rate=0.3)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    for n in (1, 31, 128, 129, 256, 257, 385, 148 * 256, 148 * 512 + 1):
        desc = edge_descriptors(centers, n, seed=n)
        same = np.repeat(desc[:1], n, axis=0)
        for d in (desc, same):
            got = _lookup(voc, d, "tensor_u8")
            want = oracle.lookup(centers, B, L, d, threads=8)
            assert np.array_equal(got, want), f"n={n}: {np.count_nonzero(got != want)} mismatches"
    assert voc.device_errors() == (0, 0)


def test_sorted_pass_with_more_tiles_than_one_round_of_ctas_holds():
    """65,536 groups and 2.8M rows: tile lists longer than one CTA per SM can hold."""
    centers, masks, weights = random_tree(16, 5, seed=5)
    voc = rbw.vocabulary_from_host(16, 5, centers, masks, weights)
    desc = torch.randint(0, 256, (2_800_003, 128), dtype=torch.uint8, device="cuda",
                         generator=torch.Generator("cuda").manual_seed(1))
    assert torch.equal(voc.lookup(desc, algo="tensor_u8"), voc.lookup(desc, algo="simt_f32"))
    assert voc.device_errors() == (0, 0)


@pytest.mark.parametrize("B,L", [(3, 8), (10, 4), (12, 4)])
def test_center_slots_used_again_and_again_hold_their_own_norms(B, L):
    """Groups of few rows: every CTA loads many center blocks into its two to four slots, over the norm
    keys of the blocks before.  Each of several lookups equals the FP32 kernel."""
    centers, masks, weights = random_tree(B, L, seed=B * L + 1, dup_rate=0.2)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = torch.randint(0, 256, (250_007, 128), dtype=torch.uint8, device="cuda",
                         generator=torch.Generator("cuda").manual_seed(B))
    want = voc.lookup(desc, algo="simt_f32")
    for _ in range(6):
        assert torch.equal(voc.lookup(desc, algo="tensor_u8"), want)
    assert voc.device_errors() == (0, 0)


def test_sorted_pass_with_more_groups_than_rows_in_several_rounds():
    """117,649 groups and 100,003 rows: nearly every super-tile holds a few rows, and they are more than
    one round of CTAs holds the lists of, by the count of groups that can have rows."""
    centers, masks, weights = random_tree(7, 7, seed=6, dup_rate=0.0)
    voc = rbw.vocabulary_from_host(7, 7, centers, masks, weights)
    g = torch.Generator("cuda").manual_seed(2)
    for n in (100_003, 75_777):
        desc = torch.randint(0, 256, (n, 128), dtype=torch.uint8, device="cuda", generator=g)
        assert torch.equal(voc.lookup(desc, algo="tensor_u8"), voc.lookup(desc, algo="simt_f32"))
    assert voc.device_errors() == (0, 0)


@pytest.mark.parametrize("algo", ["auto", "tensor_u8", "tensor_u8_ring", "simt_f32", "noalloc"])
def test_lookup_as_the_first_call_of_a_thread(oracle, algo):
    """A thread that has made no CUDA call yet looks descriptors up, on a stream of its own."""
    import threading

    B, L, n = 16, 4, 100_003
    centers, masks, weights = random_tree(B, L, seed=14)
    voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
    desc = edge_descriptors(centers, n, seed=15)
    rows, stream = torch.from_numpy(desc).cuda(), torch.cuda.Stream()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    failed = []

    def work():
        try:
            if algo == "noalloc":
                voc.lookup_noalloc(rows, out, stream=stream)
            else:
                voc.lookup(rows, out, algo=algo, stream=stream)
        except Exception as e:
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not failed, failed
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.lookup(centers, B, L, desc, threads=8))


@pytest.mark.parametrize("B,L,float_centers", [(16, 3, False), (10, 6, False), (3, 7, False), (16, 2, True), (9, 4, True)])
def test_centers_come_back_as_they_went_in(B, L, float_centers):
    """Trees above and below one 32 MiB piece of the packed copy, with and without padded slots, and
    the memory of a freed tree used again."""
    rng = np.random.default_rng(B * L)
    nodes = sum(B ** i for i in range(L))
    masks = np.full(nodes, (1 << B) - 1, np.uint32)
    weights = rng.random((nodes, B), np.float32)
    for _ in range(2):
        if float_centers:
            centers = (rng.random((nodes, B, 128), np.float32) * 255).astype(np.float32)
            voc = rbw.vocabulary_from_host_f32(B, L, centers, masks, weights)
            assert np.array_equal(voc.centers_f32(), centers)
            assert np.array_equal(voc.tree()[0], np.rint(centers).astype(np.uint8))
        else:
            centers = rng.integers(0, 256, (nodes, B, 128), dtype=np.uint8)
            voc = rbw.vocabulary_from_host(B, L, centers, masks, weights)
            assert np.array_equal(voc.tree()[0], centers)
        assert voc.device_errors() == (0, 0)
        del voc


_FULL_GPU = """
import numpy as np, torch
import rapidbow_b200 as rbw

B, L = 10, 5
nodes = sum(B ** i for i in range(L))
centers = np.random.default_rng(3).integers(0, 256, (nodes, B, 128), dtype=np.uint8)
tree = np.full(nodes, 1023, np.uint32), np.ones((nodes, B), np.float32)
voc = rbw.vocabulary_from_host(B, L, centers, *tree)
vof = rbw.vocabulary_from_host_f32(B, 3, centers[:111].astype(np.float32), tree[0][:111], tree[1][:111])
torch.cuda.synchronize()
hold, size = [], 1 << 34
while size >= 1 << 20:
    try:
        hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        size //= 2
assert np.array_equal(voc.tree()[0], centers)
assert np.array_equal(vof.centers_f32(), centers[:111].astype(np.float32))
print("read back")
"""


def test_centers_come_back_without_device_memory_to_spare():
    """Trees with padded slots are packed on the device first, and copied as they lie where the GPU's
    memory is all in use (in a process of its own, whose pool is empty)."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FULL_GPU], capture_output=True, text=True, cwd=root, timeout=300)
    assert r.returncode == 0 and "read back" in r.stdout, r.stderr
