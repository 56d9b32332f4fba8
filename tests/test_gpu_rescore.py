"""Batched tensor-core rescoring (tcgen05 kind::i8) against the int64 oracle.

Integer work, so the bar is bit-exact: every statistic and every Gram entry
equals the oracle's int64 recompute (xwo_rescore, the restatement of the
reference's rebuild_gram / verify_weighing).  At the benchmark's size (65536
matrices per order) the tensor-core results are compared with the
independent SIMT kernel for every matrix and with the oracle on a sample.
"""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O
import xtax_b200 as X

pytestmark = pytest.mark.gpu


def random_fixed_degree(count, n, w, seed):
    """Row-only fixed-degree ternary matrices: w nonzeros per row at uniform
    positions with uniform signs (row-major)."""
    rng = np.random.default_rng(seed)
    W = np.zeros((count, n, n), dtype=np.int8)
    for m in range(count):
        idx = np.argsort(rng.random((n, n)), axis=1)[:, :w]
        signs = rng.integers(0, 2, size=(n, w)) * 2 - 1
        np.put_along_axis(W[m], idx, signs.astype(np.int8), axis=1)
    return W


def oracle_stats(M, n, w):
    st, G, _ = O.rescore(n, w, M.T.reshape(-1))   # oracle takes column-major W
    exact = O.verify(n, w, M.T.reshape(-1)) == 3
    return [int(st[0]), int(st[1]), int(st[2]), 1 if (st[1] == 0 and (np.diag(G) == w).all()) else 0], G, exact


@pytest.mark.parametrize("n", [32, 64, 96, 128])
@pytest.mark.parametrize("count", [1, 3, 37, 301])
def test_tensor_core_rescore_matches_oracle(n, count):
    w = n // 2
    W = random_fixed_degree(count, n, w, seed=n * 1000 + count)
    # plant exact weighing matrices: direct sums of Sylvester blocks of order 32
    syl = O.sylvester(n, 32).reshape(n, n).T.astype(np.int8)   # row-major
    for m in range(0, count, 7):
        W[m] = syl
    stats, G = X.rescore(W, n, w, gram=True)
    for m in range(count):
        ww = 32 if m % 7 == 0 else w
        ref, Gref, _ = oracle_stats(W[m], n, ww)
        if ww != w:
            # the diagonal check uses the call's w: Sylvester rows have weight 32
            ref[3] = 1 if (ref[1] == 0 and (np.diag(Gref) == w).all()) else 0
        assert stats[m].tolist() == ref, (m, stats[m], ref)
        assert (G[m] == Gref).all(), m


@pytest.mark.parametrize("n", [32, 64, 96, 128])
def test_rescore_at_benchmark_size(n):
    torch = pytest.importorskip("torch")
    count, w = 65536, n // 2
    gen = torch.Generator(device="cuda").manual_seed(n)
    # fixed-degree rows on the device: random permutation keys pick w columns
    W = torch.zeros((count, n, n), dtype=torch.int8, device="cuda")
    for c0 in range(0, count, 4096):
        keys = torch.rand((4096, n, n), device="cuda", generator=gen)
        idx = keys.argsort(dim=2)[:, :, :w]
        signs = (torch.randint(0, 2, (4096, n, w), device="cuda", generator=gen) * 2 - 1).to(torch.int8)
        W[c0:c0 + 4096].scatter_(2, idx, signs)
        del keys, idx, signs
    s_tc = torch.zeros((count, 4), dtype=torch.int32, device="cuda")
    s_simt = torch.zeros((count, 4), dtype=torch.int32, device="cuda")
    rc = X.lib().xw_rescore_device(C.c_void_p(W.data_ptr()), count, n, w, C.c_void_p(s_tc.data_ptr()), None, 0, None)
    assert rc == X.XW_OK
    rc = X.lib().xw_rescore_device(C.c_void_p(W.data_ptr()), count, n, w, C.c_void_p(s_simt.data_ptr()), None, 1,
                                   None)
    assert rc == X.XW_OK
    torch.cuda.synchronize()
    assert X.lib().xw_rescore_status() == X.XW_OK
    assert torch.equal(s_tc, s_simt)
    Wh = W.cpu().numpy()
    sh = s_tc.cpu().numpy()
    rng = np.random.default_rng(n)
    for m in rng.choice(count, 64, replace=False):
        ref, _, _ = oracle_stats(Wh[m], n, w)
        assert sh[m].tolist() == ref, m


@pytest.mark.parametrize("n", [1, 5, 12, 26, 63, 100, 127, 160, 256])
def test_simt_rescore_for_orders_off_the_tensor_core_grid(n):
    # orders that are not multiples of 32 take the SIMT kernel
    count, w = 17, max(1, n // 3)
    W = random_fixed_degree(count, n, w, seed=500 + n)
    stats, G = X.rescore(W, n, w, gram=True)
    for m in range(count):
        ref, Gref, _ = oracle_stats(W[m], n, w)
        assert stats[m].tolist() == ref, (m, stats[m], ref)
        assert (G[m] == Gref).all(), m


def test_rescore_empty_batch_and_bad_arguments():
    import ctypes as C
    stats = np.zeros((1, 4), dtype=np.int32)
    W = np.zeros((1, 32, 32), dtype=np.int8)
    assert X.lib().xw_rescore(W.ctypes.data_as(C.POINTER(C.c_int8)), 0, 32, 16,
                              stats.ctypes.data_as(C.POINTER(C.c_int32)), None) == X.XW_OK
    assert X.lib().xw_rescore(W.ctypes.data_as(C.POINTER(C.c_int8)), 1, 257, 16,
                              stats.ctypes.data_as(C.POINTER(C.c_int32)), None) == X.XW_ERR_INVALID


@pytest.mark.parametrize("count", [1, 5, 700])
@pytest.mark.parametrize("n", [9, 13, 16, 17, 31, 33, 47, 63, 65, 95, 97, 100, 127, 129, 159, 161, 192, 193, 224, 255])
def test_padded_tensor_core_rescore_matches_int64(n, count):
    # orders off the 32-grid (padded tiles; the remainders of a 32-row block,
    # of a 16-byte chunk and of a K-half) and orders above 128: one matrix,
    # a part-filled tile, more tiles than CTAs; every value an integer
    if n > 128:
        count = min(count, 160)
    W = random_fixed_degree(count, n, max(1, (2 * n) // 3), seed=900 + n)
    W[0] = np.eye(n, dtype=np.int8)          # an exact W(n,1) among them
    w = 1
    stats, G = X.rescore(W, n, w, gram=True)
    ref = np.matmul(W.astype(np.float64), W.astype(np.float64).transpose(0, 2, 1)).astype(np.int64)
    assert (G == ref).all()
    off = ref * (1 - np.eye(n, dtype=np.int64))
    want = np.stack([np.abs(off).sum((1, 2)) // 2, (off != 0).sum((1, 2)) // 2, (off * off).sum((1, 2)) // 2,
                     (ref == w * np.eye(n, dtype=np.int64)).all((1, 2))], 1)
    assert (stats == want).all()
    assert (X.rescore(W, n, w) == want).all()


@pytest.mark.parametrize("shift", [1, 3, 8, 15])
@pytest.mark.parametrize("n", [26, 32, 64, 100, 128, 150])
def test_rescore_of_device_input_at_any_address(n, shift):
    # the input starts `shift` bytes off a 16-byte boundary and ends at the
    # end of its allocation's values
    torch = pytest.importorskip("torch")
    import ctypes as C
    count, w = 9, n // 2
    W = random_fixed_degree(count, n, w, seed=50 + n)
    buf = torch.full((W.size + shift,), 77, dtype=torch.int8, device="cuda")
    buf[shift:] = torch.from_numpy(W.reshape(-1)).cuda()
    out = torch.zeros((count, 4), dtype=torch.int32, device="cuda")
    assert X.lib().xw_rescore_device(C.c_void_p(buf.data_ptr() + shift), count, n, w, C.c_void_p(out.data_ptr()), None, 0,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream)) == X.XW_OK
    torch.cuda.synchronize()
    assert X.lib().xw_rescore_status() == X.XW_OK
    assert (out.cpu().numpy() == X.rescore(W, n, w)).all()
    for m in range(count):
        assert out[m].tolist() == oracle_stats(W[m], n, w)[0]


@pytest.mark.parametrize("top", [1, 2, 5])
@pytest.mark.parametrize("n", [32, 64, 96, 100, 128, 192])
def test_rescore_of_entries_that_do_not_fit_a_byte(n, top):
    # Gram entries of up to 128 and beyond: equal full rows (w = n) and
    # entries up to `top`, in some matrices of a batch only, so that the byte
    # form and the word form of the epilogue run side by side
    rng = np.random.default_rng(n + top)
    count = 40
    W = random_fixed_degree(count, n, n // 2, seed=n)
    for m in range(0, count, 3):
        W[m] = rng.integers(-top, top + 1, size=(n, n))
        W[m, 1] = W[m, n - 1] = top
        W[m, n // 2] = -top
    ref = np.matmul(W.astype(np.float64), W.astype(np.float64).transpose(0, 2, 1)).astype(np.int64)
    off = ref * (1 - np.eye(n, dtype=np.int64))
    want = np.stack([np.abs(off).sum((1, 2)) // 2, (off != 0).sum((1, 2)) // 2, (off * off).sum((1, 2)) // 2,
                     np.zeros(count, dtype=np.int64)], 1)
    assert want.max() < 2 ** 30   # twice the squared score is summed in 32 bits
    assert (X.rescore(W, n, n // 2) == want).all()


@pytest.mark.parametrize("n", [128, 216, 256])
def test_rescore_of_equal_full_rows(n):
    # every Gram entry is +-n: the largest squared score of ternary
    # matrices, twice which passes 2^31 from n = 216 on
    W = np.ones((3, n, n), dtype=np.int8)
    W[1, ::2] = -1
    want = [n * (n - 1) // 2 * n, n * (n - 1) // 2, n * (n - 1) // 2 * n * n, 0]
    assert want[2] < 2 ** 31
    stats, G = X.rescore(W, n, n, gram=True)
    assert (np.abs(G) == n).all()
    assert stats.tolist() == [want] * 3
    assert X.rescore(W, n, n).tolist() == [want] * 3
    torch = pytest.importorskip("torch")
    import ctypes as C
    d, out = torch.from_numpy(W).cuda(), torch.zeros((3, 4), dtype=torch.int32, device="cuda")
    assert X.lib().xw_rescore_device(C.c_void_p(d.data_ptr()), 3, n, n, C.c_void_p(out.data_ptr()), None, 1,
                                     None) == X.XW_OK
    torch.cuda.synchronize()
    assert out.tolist() == [want] * 3


@pytest.mark.parametrize("n,count", [(9, 3999), (9, 7999), (9, 8000), (10, 3999), (10, 4000), (12, 4000)])
def test_rescore_on_both_sides_of_the_tiny_orders_line(n, count):
    W = random_fixed_degree(40, n, n - 1, seed=n).repeat((count + 39) // 40, axis=0)[:count]
    W[count - 1] = np.eye(n, dtype=np.int8)
    ref = np.matmul(W.astype(np.int64), W.astype(np.int64).transpose(0, 2, 1))
    off = ref * (1 - np.eye(n, dtype=np.int64))
    want = np.stack([np.abs(off).sum((1, 2)) // 2, (off != 0).sum((1, 2)) // 2, (off * off).sum((1, 2)) // 2,
                     (ref == np.eye(n, dtype=np.int64)).all((1, 2))], 1)
    assert (X.rescore(W, n, 1) == want).all()
