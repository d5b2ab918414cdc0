"""GPU parity at the edges of the tiles, chunks and clusters of the kernels that products, triangular solves
and poolings are dispatched to by size, type and alignment, against the oracle with a double accumulator."""
import numpy as np
import pytest
import torch

import oracle
from support import max_rel, rel_fro

pytestmark = pytest.mark.gpu

FP32_TOL = 1e-5
HALF_TOL = 2e-2


@pytest.fixture(scope="module")
def lib():
    import dlf_b200
    return dlf_b200


@pytest.fixture(autouse=True)
def _device_status_clean(lib):
    yield
    lib.set_tuning(0, 0)
    assert lib.device_status() == 0, "a device-side bounded wait timed out"


def _round_to(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(dtype).float().numpy()


def _close(got, ref, dtype):
    if dtype == torch.float32:
        return rel_fro(got, ref) <= FP32_TOL
    return max_rel(got, ref) <= HALF_TOL


def _gemm_against_oracle(dtype, m, n, k, ta, tb, alpha, beta, pad, offset, seed):
    """One row-major call on matrices whose lines are `pad` elements longer than needed and start `offset`
    elements into their buffers; also checks that nothing outside the m x n window changes."""
    from dlf_b200 import gblas as gb
    rng = np.random.default_rng(seed)
    lda, ldb, ldc = (m if ta else k) + pad, (k if tb else n) + pad, n + pad
    A = _round_to(rng.uniform(-1, 1, offset + (k if ta else m) * lda), dtype)
    B = _round_to(rng.uniform(-1, 1, offset + (n if tb else k) * ldb), dtype)
    C = _round_to(rng.normal(size=offset + m * ldc + 16), dtype)
    TA, TB = (gb.Transpose.Trans if t else gb.Transpose.NoTrans for t in (ta, tb))
    ref = C.copy()
    oracle.gblas_sgemm(oracle.ROW_MAJOR, int(TA), int(TB), m, n, k, alpha, A, offset, lda, B, offset, ldb, beta, ref, offset, ldc, wide=True)
    start = C.copy()
    window = np.zeros(C.size, dtype=bool)
    window[offset:offset + m * ldc].reshape(m, ldc)[:, :n] = True
    if beta == 0:
        start[window] = np.nan  # must not be read
    c = torch.from_numpy(start).to(dtype).cuda()
    gb.gemm(gb.Layout.RowMajor, TA, TB, m, n, k, alpha, torch.from_numpy(A).to(dtype).cuda(), offset, lda,
            torch.from_numpy(B).to(dtype).cuda(), offset, ldb, beta, c, offset, ldc)
    got = c.float().cpu().numpy()
    assert np.array_equal(got[~window], start[~window])
    assert _close(got[window], ref[window], dtype), (m, n, k, ta, tb, alpha, beta)


@pytest.mark.parametrize("width", [0, 64, 128, 192])
@pytest.mark.parametrize("m,n,k", [
    (4, 8, 4),          # one partly filled tile, less than a k-block
    (129, 132, 260),    # a row and four columns into the next tile, a ninth k-block: a second chunk of one
    (196, 260, 256),    # exactly one chunk
    (68, 196, 1028),    # clusters: the last CTA's share is longer
])
def test_fp32_products_through_tensor_maps(lib, width, m, n, k):
    """contraction_f32_kernel at every tile width, all transposes, with and without beta."""
    lib.set_tuning(width, 0)
    for ta in (False, True):
        for tb in (False, True):
            _gemm_against_oracle(torch.float32, m, 4 * ((n + 3) // 4), k, ta, tb, 1.0, 0.0, 0, 0, m + n + k)
            _gemm_against_oracle(torch.float32, 4 * ((m + 3) // 4), 4 * ((n + 3) // 4), k, ta, tb, 0.5, 0.25, 4, 4, m + n + k + 1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [
    (8, 8, 8),          # one CTA, one k-block
    (129, 72, 504),     # tile edges, seven k-blocks: not split
    (130, 72, 520),     # nine k-blocks over two CTAs
    (64, 2056, 1032),   # 33 tiles of 17 k-blocks over four
    (1000, 328, 2056),  # 33 k-blocks; more than 16 tiles
])
def test_16_bit_products_shared_by_a_cluster(lib, dtype, m, n, k):
    """contraction_split_kernel: row and column remainders, uneven shares of the k-blocks, beta and alpha."""
    for ta in (False, True):
        for tb in (False, True):
            m8 = (m + 7) // 8 * 8 if ta else m
            _gemm_against_oracle(dtype, m8, n, k, ta, tb, 1.0, 0.0, 0, 0, m + n + k)
            _gemm_against_oracle(dtype, m8, n, k, ta, tb, 0.5, 0.25, 8, 8, m + n + k + 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16], ids=["f32", "f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [(129, 131, 515), (7, 1031, 1027), (333, 111, 2049)])
def test_products_of_operands_off_16_byte_boundaries(lib, dtype, m, n, k):
    """Odd leading dimensions and offsets: the operands are copied with aligned lines first
    (pad_lines_kernel); one operand aligned and the other not; offsets of every residue."""
    for ta in (False, True):
        for tb in (False, True):
            for pad, offset in ((0, 0), (1, 1), (2, 3), (3, 6)):
                _gemm_against_oracle(dtype, m, n, k, ta, tb, 1.0, 0.0, pad, offset, m + n + k)
    _gemm_against_oracle(dtype, m + 8 - m % 8, n, k, True, False, 0.5, 0.25, 0, 0, m + n + k)


def test_a_products_scratch_covers_its_aligned_copies(lib):
    """dlf_b200_gemm_scratch_bytes is dlf_b200_gemm_workspace_bytes plus the copies a call needs. With that much the copies
    are a launch of their own; with too little for them, or nothing, the same call runs in one launch."""
    import ctypes
    L = lib.lib()
    m, n, k = 150, 160, 512
    g = torch.Generator().manual_seed(4)
    a = (torch.rand(m * k + 1, generator=g) - 0.5).half().cuda()
    b = (torch.rand(k * n, generator=g) - 0.5).half().cuda()
    common = (16, 101, 111, 111, m, n, k)
    base = L.dlf_b200_gemm_workspace_bytes(16, m, n, k)
    assert L.dlf_b200_gemm_scratch_bytes(*common, a.data_ptr(), k, b.data_ptr(), n) == base
    more = L.dlf_b200_gemm_scratch_bytes(*common, a.data_ptr() + 2, k, b.data_ptr(), n)
    assert more >= base + m * k * 2
    want = (a[1:].double().view(m, k) @ b.double().view(k, n)).flatten().cpu().numpy()
    one, zero = ctypes.c_uint16(0x3C00), ctypes.c_uint16(0)
    ws = torch.empty(more, dtype=torch.uint8, device="cuda")
    launches = {}
    for nbytes in (0, m * k, more):
        c = torch.zeros(m * n, dtype=torch.float16, device="cuda")
        before = lib.launch_count()
        assert L.dlf_b200_gemm_ex(*common, ctypes.byref(one), a.data_ptr() + 2, k, b.data_ptr(), n, ctypes.byref(zero), c.data_ptr(), n,
                                  ws.data_ptr() if nbytes else None, nbytes, torch.cuda.current_stream().cuda_stream) == 0
        launches[nbytes] = lib.launch_count() - before
        assert max_rel(c.float().cpu().numpy(), want) <= HALF_TOL
    assert launches[0] == launches[m * k] == 1 and launches[more] > 1


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32], ids=["f16", "f32"])
@pytest.mark.parametrize("k", [128, 2048], ids=["one CTA", "a cluster"])
def test_waits_that_run_out_in_kernels_whose_tiles_a_cluster_may_share(lib, dtype, k):
    """The bounded waits of contraction_split_kernel and contraction_f32_kernel, made to run out once: with the test aid
    0x30000000 a single-tile launch withholds the commit that hands the accumulator on and waits about a millisecond. Every CTA
    of the cluster leaves, the status reports the time-out once, C keeps its contents, the next call is right."""
    from dlf_b200 import gblas as gb
    m, n = 64, 64
    g = torch.Generator().manual_seed(8)
    A, B = ((torch.rand(s, generator=g) * 2 - 1).to(dtype).cuda() for s in (m * k, k * n))
    C = torch.full((m * n,), 5.0, dtype=dtype, device="cuda")

    def product():
        gb.gemm(gb.Layout.RowMajor, gb.Transpose.NoTrans, gb.Transpose.NoTrans, m, n, k, 1.0, A, 0, k, B, 0, n, 0.0, C, 0, n)
        torch.cuda.synchronize()

    lib.set_tuning(0, 0x30000000)
    try:
        product()
    finally:
        lib.set_tuning(0, 0)
    assert lib.device_status() == 1
    assert lib.device_status() == 0
    assert bool((C == 5.0).all())
    product()
    ref = (A.double().view(m, k) @ B.double().view(k, n)).flatten().cpu().numpy()
    assert _close(C.float().cpu().numpy(), ref, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("q,systems", [(1, 1), (31, 5), (32, 3), (33, 600), (64, 4), (97, 1200), (448, 2400), (1024, 6), (1025, 5),
                                       # a thread per system: from 25 q^2 on, up to 32 and up to 64 unknowns
                                       (1, 25), (8, 1599), (8, 1600), (32, 25601), (33, 27300),
                                       # CTAs of 128 and 256 threads: more than 24 systems for each SM
                                       (33, 3553), (128, 3570), (129, 3553), (256, 3600),
                                       # many systems: blocks of 128 unknowns
                                       (128, 16384), (160, 16400), (300, 16384)])
def test_triangular_solves_at_the_edges_of_their_blocks(lib, dtype, q, systems):
    """l3_trsm_kernel: partly filled blocks of 32 unknowns, each number of systems per CTA, both contiguous
    directions, both substitution orders, the largest order of one launch and one more."""
    from dlf_b200 import gblas as gb
    rng = np.random.default_rng(q + systems)
    for side in (gb.Side.Left, gb.Side.Right):
        m, n = (q, systems) if side == gb.Side.Left else (systems, q)
        for tri in (gb.Triangle.Upper, gb.Triangle.Lower):
            for ta in (gb.Transpose.NoTrans, gb.Transpose.Trans):
                lda, ldb = q + 1, n + 3
                A = (0.5 / np.sqrt(q)) * rng.uniform(-1, 1, (q, lda)).astype(np.float32)
                A[np.arange(q), np.arange(q)] = rng.uniform(1.0, 2.0, q).astype(np.float32)
                A = _round_to(A, dtype)
                ii, jj = np.indices(A.shape)
                keep = (jj < q) & ((ii <= jj) if tri == gb.Triangle.Upper else (ii >= jj))
                B = _round_to(rng.uniform(-1, 1, m * ldb), dtype)
                ref = B.copy()
                oracle.trsm(int(side), int(tri), int(ta), int(gb.Diagonal.NonUnit), m, n, 0.5,
                            np.where(keep, A, 0.0).astype(np.float32).ravel(), lda, ref, ldb, wide=True)
                got = torch.from_numpy(B.copy()).to(dtype).cuda()
                gb.trsm(gb.Layout.RowMajor, side, tri, ta, gb.Diagonal.NonUnit, m, n, 0.5,
                        torch.from_numpy(np.where(keep, A, np.nan).astype(np.float32).ravel()).to(dtype).cuda(), 0, lda, got, 0, ldb)
                g = got.float().cpu().numpy()
                if dtype == torch.float32:
                    assert rel_fro(g, ref) <= FP32_TOL, (side, tri, ta)
                else:
                    assert max_rel(g, ref) <= 5e-2, (side, tri, ta)


@pytest.mark.parametrize("systems", [3, 1300, 3600, 40000], ids=["shuffles", "lane per system", "short CTAs", "thread per system"])
def test_triangular_solve_with_a_zero_and_an_infinite_pivot(lib, systems):
    """What IEEE division gives: x / 0 = inf, 0 / 0 = NaN, x / inf = 0, and nothing spreads backwards."""
    from dlf_b200 import gblas as gb
    n = 40
    T = torch.eye(n, device="cuda")
    T[2, 2], T[5, 5], T[36, 36] = float("inf"), 0.0, 2.0
    B = torch.ones(n, systems, device="cuda")
    B[5, 1] = 0.0
    gb.trsm(gb.Layout.RowMajor, gb.Side.Left, gb.Triangle.Lower, gb.Transpose.NoTrans, gb.Diagonal.NonUnit, n, systems, 1.0,
            T.view(-1), 0, n, B.view(-1), 0, systems)
    got = B.cpu()
    expected = torch.ones(5, systems)
    expected[2] = 0.0
    assert torch.equal(got[:5], expected)
    assert bool(torch.isinf(got[5, [0, 2]]).all()) and bool(torch.isnan(got[5, 1]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("shape", [(1, 2048, 7, 7), (3, 8, 2, 4), (2, 264, 3, 3), (2, 40, 33, 5), (1100, 8, 2, 4), (1500, 8, 2, 4)])
def test_global_pooling_between_channels_last_tensors(lib, dtype, shape):
    """pool_nhwc_global_kernel: channel groups that do not fill a warp, more and fewer pixels than warps; on
    either side of the number of images from which a thread walks each of them instead."""
    from dlf_b200 import gdnn
    n, c, h, w = shape
    X = _round_to(np.random.default_rng(c).normal(size=shape), dtype)
    Xn = torch.from_numpy(X).to(dtype).cuda().permute(0, 2, 3, 1).contiguous()
    for average in (True, False):
        Y = torch.empty((n, 1, 1, c), dtype=dtype, device="cuda")
        gdnn.pool_nhwc(Xn, Y, gdnn.Filter2D(shape, h, w).strides(h, w), average=average)
        got = Y.float().cpu().numpy().reshape(n, c)
        ref = oracle.global_pool(X, "avg" if average else "max", wide=True).reshape(n, c)
        if average:
            assert max_rel(got, ref) <= HALF_TOL
        else:
            assert np.array_equal(got, ref)


# the NaN that CUDA arithmetic returns, the same with a sign, numpy's, one whose payload a truncation to tf32 drops
NAN_BITS = [0x7fffffff, 0xffffffff, 0x7fc00000, 0x7f800001]


def _nan(bits):
    return np.array([bits], dtype=np.uint32).view(np.float32)[0]


@pytest.mark.parametrize("bits", NAN_BITS, ids=hex)
@pytest.mark.parametrize("width,m,n,k", [(64, 196, 260, 320), (128, 196, 260, 320), (192, 196, 260, 320), (0, 68, 196, 1028)])
def test_nan_in_a_fp32_operand_stays_nan(lib, bits, width, m, n, k):
    """contraction_f32_kernel, each tile width and tiles shared by a cluster: a NaN of any payload in either operand
    reaches every output it contributes to, and no other."""
    from dlf_b200 import gblas as gb
    rng = np.random.default_rng(m + n + k)
    lib.set_tuning(width, 0)
    for ta in (False, True):
        for tb in (False, True):
            for side in "AB":
                A = rng.uniform(-1, 1, (m, k)).astype(np.float32)
                B = rng.uniform(-1, 1, (k, n)).astype(np.float32)
                expected = np.zeros((m, n), dtype=bool)
                if side == "A":
                    A[5, 3] = A[130 % m, k - 1] = _nan(bits)
                    expected[[5, 130 % m]] = True
                else:
                    B[3, 5] = B[k - 1, 130] = _nan(bits)
                    expected[:, [5, 130]] = True
                C = torch.zeros(m * n, device="cuda")
                gb.gemm(gb.Layout.RowMajor, gb.Transpose.Trans if ta else gb.Transpose.NoTrans,
                        gb.Transpose.Trans if tb else gb.Transpose.NoTrans, m, n, k, 1.0,
                        torch.from_numpy(np.ascontiguousarray(A.T if ta else A)).cuda().view(-1), 0, m if ta else k,
                        torch.from_numpy(np.ascontiguousarray(B.T if tb else B)).cuda().view(-1), 0, k if tb else n, 0.0, C, 0, n)
                got = C.cpu().numpy().reshape(m, n)
                assert np.array_equal(np.isnan(got), expected), (ta, tb, side)
                ref = np.where(np.isnan(A), 0.0, A).astype(np.float64) @ np.where(np.isnan(B), 0.0, B).astype(np.float64)
                assert rel_fro(got[~expected], ref[~expected]) <= FP32_TOL


@pytest.mark.parametrize("bits", NAN_BITS, ids=hex)
def test_nan_in_a_stack_of_fp32_products_stays_nan(lib, bits):
    from dlf_b200 import tensor
    A, B = torch.ones(3, 132, 64), torch.ones(3, 64, 68)
    A.numpy()[1, 7, 9] = _nan(bits)
    B.numpy()[2, 9, 65] = _nan(bits)
    got = torch.isnan(tensor.matmul(A.cuda(), B.cuda(), torch.empty(3, 132, 68, device="cuda")).cpu())
    expected = torch.zeros(3, 132, 68, dtype=torch.bool)
    expected[1, 7] = True
    expected[2, :, 65] = True
    assert torch.equal(got, expected)


@pytest.mark.parametrize("bits", NAN_BITS, ids=hex)
@pytest.mark.parametrize("size,stride", [(8, 1), (7, 1), (8, 2)], ids=["planes of 16 bytes", "odd planes", "stride 2"])
def test_nan_in_a_pointwise_fp32_convolution_stays_nan(lib, bits, size, stride):
    """1x1 filters: a NaN pixel reaches that pixel of every channel, a NaN weight every pixel of its channel."""
    from dlf_b200 import gdnn
    f = gdnn.Filter2D((2, 72, size, size), (68, 72, 1, 1)).strides(stride, stride)
    X, W = torch.ones(2, 72, size, size), torch.ones(68, 72, 1, 1)
    X.numpy()[1, 70, 4, 6] = _nan(bits)
    W.numpy()[66, 71] = _nan(bits)
    Y = torch.empty(f.output_shape(), device="cuda")
    gdnn.conv2d_filter(X.cuda(), W.cuda(), Y, f)
    expected = torch.zeros(f.output_shape(), dtype=torch.bool)
    expected[1, :, 4 // stride, 6 // stride] = True
    expected[:, 66] = True
    assert torch.equal(torch.isnan(Y.cpu()), expected)


def test_unaligned_products_from_two_threads_on_one_stream(lib):
    """Each call queues copies of its operands and a product that reads them, in scratch the stream's calls share."""
    import threading
    from dlf_b200 import tensor
    g = torch.Generator().manual_seed(5)
    operands = [(torch.rand(601, 515 + 2 * i, generator=g).cuda(), torch.rand(515 + 2 * i, 803, generator=g).cuda()) for i in range(2)]
    wanted = [(a.double() @ b.double()).float() for a, b in operands]
    results = [[torch.empty(601, 803, device="cuda") for _ in range(300)] for _ in range(2)]
    torch.cuda.synchronize()

    def work(i):
        for y in results[i]:
            tensor.matmul(*operands[i], y)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        for y in results[i]:
            assert float((y - wanted[i]).norm() / wanted[i].norm()) <= FP32_TOL


def test_a_captured_unaligned_product_survives_larger_ones(lib):
    """The scratch of a captured call belongs to its graph: later calls on the stream that need more of it must
    not take away what the replays write."""
    from dlf_b200 import tensor
    g = torch.Generator().manual_seed(6)

    def operands(m, n, k):
        a, b = torch.rand(m, k, generator=g).cuda(), torch.rand(k, n, generator=g).cuda()
        return a, b, torch.empty(m, n, device="cuda")

    a, b, y = operands(601, 803, 515)
    tensor.matmul(a, b, y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tensor.matmul(a, b, y)
    large = operands(1601, 1603, 1605)
    tensor.matmul(*large)
    others = [torch.full((601 * 516 * 4,), 7, dtype=torch.uint8, device="cuda") for _ in range(16)]
    y.zero_()
    graph.replay()
    assert float((y - a @ b).norm() / y.norm()) <= 2e-3  # (torch's product of fp32 matrices may use tf32)
    assert all(bool((o == 7).all()) for o in others)


@pytest.mark.parametrize("size,stride", [(8, 1), (7, 1), (14, 2)], ids=["planes of 16 bytes", "odd planes", "stride 2"])
@pytest.mark.parametrize("channels,filters", [(48, 64), (48, 200)])
def test_pointwise_fp32_filters_keep_all_but_the_last_bit(lib, channels, filters, size, stride):
    """A 1x1 filter bank over pixels that are one in one channel each: what comes out are the weights as the kernel
    holds them. Rounded to tf32 (11 bits), the rest rounded to tf32 again: within 2^-23 of the value."""
    from dlf_b200 import gdnn
    rng = np.random.default_rng(filters)
    f = gdnn.Filter2D((1, channels, size, size), (filters, channels, 1, 1)).strides(stride, stride)
    pixels = f.output_h * f.output_w
    assert pixels >= channels
    X = np.zeros((channels, size, size), np.float32)
    kept = X[:, ::stride, ::stride]
    for c in range(channels):
        kept[c, c // f.output_w, c % f.output_w] = 1.0
    W = rng.normal(size=(filters, channels)).astype(np.float32)
    Y = torch.empty(f.output_shape(), device="cuda")
    gdnn.conv2d_filter(torch.from_numpy(X).cuda(), torch.from_numpy(W).cuda(), Y, f)
    got = Y.cpu().numpy().reshape(filters, pixels)[:, :channels]
    assert (np.abs(got.astype(np.float64) - W) <= 2.0 ** -23 * np.abs(W)).all()


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_copied_fp32_operands_keep_all_but_the_last_bit(lib, ta, tb):
    """Operands off 16-byte boundaries times the identity: within 2^-23 of the value, on either side."""
    from dlf_b200 import tensor
    rng = np.random.default_rng(3)
    n = 261
    for first in (True, False):
        M = torch.from_numpy(rng.normal(size=(n, n)).astype(np.float32)).cuda()
        I = torch.eye(n, device="cuda")
        A, B = (M, I) if first else (I, M)
        got = tensor.matmul(A.t() if ta else A, B.t() if tb else B, torch.empty(n, n, device="cuda"))
        want = M.t() if (ta if first else tb) else M
        assert bool(((got.double() - want.double()).abs() <= 2.0 ** -23 * want.double().abs()).all())


@pytest.mark.parametrize("scratch", [True, False], ids=["scratch", "no scratch"])
@pytest.mark.parametrize("n,c,h,w,k,stride", [
    (150, 4, 4, 4, 8, 1),       # gathered: little but output to write
    (140, 4, 4, 4, 8, 1),       # ... all tiles at once: a product per image
    (160, 8, 4, 4, 8, 1),       # an eighth of the rows in use: copied
    (200, 12, 10, 10, 20, 1),   # three quarters and a bit: a product per image
    (200, 12, 8, 11, 16, 1),    # less: copied
    (3, 100, 7, 9, 132, 1),     # odd planes
    (5, 36, 9, 8, 260, 2),      # stride 2
    (110, 264, 13, 13, 8, 1),   # gathered, nine k-blocks: a second chunk of one
    (98, 512, 14, 14, 24, 1),   # a product per image, two waves of tiles: split filters
    (300, 40, 9, 9, 68, 1),     # copied, two waves of tiles: split filters
])
def test_pointwise_fp32_convolutions_on_every_route(lib, n, c, h, w, k, stride, scratch):
    """Each kernel that a 1x1 filter may go to, with the scratch it asks for and without any; bias, residual, ReLU."""
    from dlf_b200 import gdnn
    rng = np.random.default_rng(n + c)
    f = gdnn.Filter2D((n, c, h, w), (k, c, 1, 1)).strides(stride, stride)
    X, W = rng.normal(size=(n, c, h, w)).astype(np.float32), (rng.normal(size=(k, c, 1, 1)) / np.sqrt(c)).astype(np.float32)
    b, R = rng.normal(size=k).astype(np.float32), rng.normal(size=f.output_shape()).astype(np.float32)
    x, wt, bt, r = (torch.from_numpy(t).cuda() for t in (X, W, b, R))
    Y = torch.full(f.output_shape(), float("nan"), device="cuda")
    if scratch:
        gdnn.conv2d_filter(x, wt, Y, f, bias=bt, residual=r, activation="relu")
    else:
        rc = lib.lib().dlf_b200_conv2d_fused(
            32, n, c, h, w, f.output_h, f.output_w, k, 1, 1, 1, 0, 0, 0, 0, stride, stride, 1, 1, x.data_ptr(), wt.data_ptr(),
            bt.data_ptr(), r.data_ptr(), 1, Y.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream)
        assert rc == 0
    want = np.einsum("oc,nchw->nohw", W[:, :, 0, 0].astype(np.float64), X[:, :, ::stride, ::stride].astype(np.float64))
    want = np.maximum(want + b[None, :, None, None] + R, 0.0)
    # chunks of 256 k on every route: 1.8e-6 of the sums (in one chunk, 512 k: 3.6e-6)
    assert rel_fro(Y.cpu().numpy(), want) <= 2.4e-6


def test_triangular_solves_of_different_orders_from_two_threads(lib):
    """Solves of order 1024 on one thread's stream and of order 48 on another's: the same kernel with much and with
    little shared memory. Every call is accepted, and the last results are right."""
    import ctypes
    import threading
    from dlf_b200 import gblas as gb
    one = ctypes.c_float(1.0)
    problems, failures = [], []
    for q in (1024, 48):
        g = torch.Generator(device="cuda").manual_seed(q)
        T = torch.randn(q, q, generator=g, device="cuda") * (0.5 / q ** 0.5)
        T.diagonal().abs_().add_(1.0)
        B = torch.randn(q, 64, generator=g, device="cuda")
        want = torch.linalg.solve_triangular(torch.tril(T).double(), B.double(), upper=False).cpu().numpy()
        problems.append((q, T, B, B.clone(), torch.cuda.Stream(), want))
    torch.cuda.synchronize()

    def work(q, T, B, X, stream, want):
        args = [32, gb.Layout.RowMajor, gb.Side.Left, gb.Triangle.Lower, gb.Transpose.NoTrans, gb.Diagonal.NonUnit, q, 64,
                ctypes.byref(one), T.data_ptr(), q, X.data_ptr(), 64, None, 0, stream.cuda_stream]
        trsm = lib.lib().dlf_b200_trsm
        for _ in range(3000):
            rc = trsm(*args)
            if rc != 0:
                failures.append((q, rc))
        with torch.cuda.stream(stream):
            X.copy_(B)
            failures.extend((q, rc) for rc in [trsm(*args)] if rc != 0)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=p) for p in problems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    for q, T, B, X, stream, want in problems:
        assert rel_fro(X.cpu().numpy(), want) <= FP32_TOL


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("m,n,k", [
    (136, 2304, 2048),   # 36 tiles of 128 x 128: a cluster of two for each tile of 128 x 64
    (640, 1024, 1024),   # 40: one CTA a tile
    (640, 1024, 8192),   # ... and so many k-blocks that they are cut into slices
    (16, 4096, 8192),    # 32 tiles of few rows, sliced
    (72, 1024, 256),     # one CTA a tile of the cluster kernel, few rows
])
def test_16_bit_products_in_one_launch_or_in_slices(lib, dtype, m, n, k):
    """Either side of the rule that cuts a product's K range between the CTAs of a cluster or between launches."""
    from dlf_b200 import tensor
    g = torch.Generator().manual_seed(k)
    A, B = (torch.rand(m, k, generator=g) - 0.5).to(dtype).cuda(), (torch.rand(k, n, generator=g) - 0.5).to(dtype).cuda()
    got = tensor.matmul(A, B, torch.empty(m, n, dtype=dtype, device="cuda"))
    assert max_rel(got.float().cpu().numpy(), (A.double() @ B.double()).cpu().numpy()) <= HALF_TOL


def test_a_forward_of_clusters_and_dependent_launches_repeats_itself(lib):
    """Partial tiles are added in rank order and dependent launches wait for what they read: the same bits every time."""
    from dlf_b200 import gdnn
    g = torch.Generator().manual_seed(2)
    X = (torch.rand(1, 14, 14, 256, generator=g) - 0.5).half().cuda()
    f = gdnn.Filter2D((1, 256, 14, 14), (256, 256, 3, 3)).pads(1, 1)
    W = [gdnn.pack_filters_nhwc(((torch.rand(256, 256, 3, 3, generator=g) - 0.5) / 16).half().cuda()) for _ in range(4)]
    first = None
    for _ in range(50):
        x = X
        for w in W:
            y = torch.empty_like(X)
            gdnn.conv2d_nhwc(x, w, y, f, residual=X, activation="relu")
            x = y
        if first is None:
            first = x
        assert torch.equal(x, first)
