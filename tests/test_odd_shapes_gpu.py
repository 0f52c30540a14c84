"""Tensor-core paths at shapes that are no multiple of a tile: strided convolutions (residue classes of the input gradient, classes no
tap reaches), channel counts that are no multiple of 32, matrices whose rows are no whole 16-byte pieces, an odd number of images
under split operands.  Oracle in float64; tolerances per math mode as in test_abi_gpu.py."""
import numpy as np
import pytest

from oracle import nocta_oracle as O
from tests.test_abi_gpu import MODE_3X, MODE_RNA, MODE_TF32, P, TOL_3X, TOL_F32, TOL_TF32, _release_uploads, abi, close, dev, host, ok  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
MODES = [(MODE_TF32, TOL_TF32), (MODE_RNA, TOL_TF32), (MODE_3X, TOL_3X)]


@pytest.fixture(autouse=True)
def _plain_f32_outputs(abi):  # noqa: F811
    abi.nc_cuda_set_round_outputs(0)


# N, Cin, H, W, Cout, k, stride, pad
CONV = [
    (3, 32, 15, 17, 64, 3, 2, 1),    # odd extents: the residue classes differ in size
    (2, 64, 28, 28, 128, 3, 2, 1),
    (3, 20, 13, 9, 36, 3, 2, 0),     # channels no multiple of 32, no padding
    (2, 32, 16, 16, 32, 1, 2, 0),    # 1 x 1: three of four classes have no tap, their gradient is zero
    (2, 48, 20, 22, 40, 5, 2, 2),
    (5, 32, 12, 12, 160, 2, 2, 0),   # every class has one tap
    (3, 48, 44, 44, 48, 3, 1, 1),    # halo kernels, pixels on M with 48 of 64 columns; odd image count
    (3, 48, 40, 26, 96, 3, 1, 1),
    (3, 96, 25, 33, 192, 3, 1, 1),   # channels on M, 64 of the second 128 rows; weight gradient in 96-column tiles
    (3, 20, 24, 24, 36, 3, 1, 1),
    (1, 36, 70, 66, 100, 3, 1, 1),
    (5, 192, 11, 11, 192, 3, 1, 1),  # low images: per-tap kernel
    (3, 40, 11, 13, 24, 3, 1, 1),
    (2, 32, 14, 15, 32, 9, 1, 4),    # more than 64 taps
]


@pytest.mark.parametrize("mode,tol", MODES)
@pytest.mark.parametrize("case", CONV)
def test_conv_odd(abi, mode, tol, case):  # noqa: F811
    from nocta_b200.cuda_abi import size4
    N, Ci, H, W, Co, k, s, p = case
    rng = np.random.default_rng(sum(case))
    x, w = rng.standard_normal((N, Ci, H, W)).astype(np.float32), (rng.standard_normal((Co, Ci, k, k)) / np.sqrt(Ci * k * k)).astype(np.float32)
    b = rng.standard_normal(Co).astype(np.float32)
    yo = O.conv2d_forward(x, w, b, s, p)
    Ho, Wo = yo.shape[2:]
    g = rng.standard_normal(yo.shape).astype(np.float32)
    dxo, dwo, dbo = O.conv2d_backward(x, w, g, s, p)
    abi.nc_cuda_set_math_mode(mode)
    put = lambda a: dev(a.transpose(0, 2, 3, 1))  # noqa: E731
    get = lambda t, sh: host(t).reshape(sh[0], sh[2], sh[3], sh[1]).transpose(0, 3, 1, 2)  # noqa: E731
    xs, ys = size4([H * W * Ci, 1, W * Ci, Ci]), size4([Ho * Wo * Co, 1, Wo * Co, Co])
    nan = lambda n: torch.full((n,), float("nan"), device="cuda")  # noqa: E731
    y, gx, gw, gb = nan(yo.size), nan(x.size), nan(w.size), nan(Co)
    tx, tg, tw = put(x), put(g), dev(w)
    ok(abi, abi.nc_cuda_conv2d_forward_f32_ex(P(y), ys, P(tx), xs, P(tw), P(dev(b)), N, Ci, H, W, Co, k, k, s, p, None))
    ok(abi, abi.nc_cuda_conv2d_backward_weight_f32_ex(P(gw), P(gb), P(tg), ys, P(tx), xs, N, Ci, H, W, Co, k, k, s, p, None))
    ok(abi, abi.nc_cuda_conv2d_backward_input_f32_ex(P(gx), xs, P(tg), ys, P(tw), N, Ci, H, W, Co, k, k, s, p, None))
    close(get(y, yo.shape), yo, tol)
    close(get(gx, x.shape), dxo, tol)
    close(host(gw).reshape(w.shape), dwo, tol)
    close(host(gb), dbo, TOL_F32)


# rows, inputs, outputs: leading dimensions of 4n + 1, 2, 3; one side aligned; several tiles with remainders; a split reduction
@pytest.mark.parametrize("mode,tol", MODES)
@pytest.mark.parametrize("B,I,Oo", [(300, 310, 250), (257, 1025, 131), (1001, 310, 1250), (130, 512, 383), (129, 515, 512), (300, 4096, 35)])
def test_linear_odd(abi, mode, tol, B, I, Oo):  # noqa: F811
    rng = np.random.default_rng(B + I + Oo)
    x, W = rng.standard_normal((B, I)).astype(np.float32), (rng.standard_normal((Oo, I)) / np.sqrt(I)).astype(np.float32)
    b, g = rng.standard_normal(Oo).astype(np.float32), rng.standard_normal((B, Oo)).astype(np.float32)
    abi.nc_cuda_set_math_mode(mode)
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")  # noqa: E731
    y, gx, gW, gb = nan(B, Oo), nan(B, I), nan(Oo, I), nan(Oo)
    tx, tW, tg = dev(x), dev(W), dev(g)
    ok(abi, abi.nc_cuda_linear_forward_f32_ex(P(y), P(tx), P(tW), P(dev(b)), B, I, Oo, None))
    ok(abi, abi.nc_cuda_linear_backward_f32_ex(P(gx), P(gW), P(gb), P(tg), P(tx), P(tW), B, I, Oo, None))
    dx, dW, db = O.linear_backward(g, x, W)
    close(host(y), O.linear_forward(x, W, b), tol)
    close(host(gx), dx, tol)
    close(host(gW), dW, tol)
    close(host(gb), db, TOL_F32)


# products that fill the chip without a split reduction: 256 x 256 tiles of SM pairs with remainders in rows, columns (also ones whose
# output rows are no whole 16-byte pieces) and reduction, one tile and several per pair, every operand order, alpha and beta
@pytest.mark.parametrize("M,N,K,ta,tb", [(2561, 1024, 160, 0, 1), (2500, 1030, 196, 0, 1), (2080, 1056, 132, 1, 0), (2464, 1088, 1000, 0, 0),
                                         (1056, 2500, 256, 1, 1), (4999, 2052, 128, 0, 1)])
def test_large_products(abi, M, N, K, ta, tb):  # noqa: F811
    rng = np.random.default_rng(M + N + K)
    A, B = rng.standard_normal((K, M) if ta else (M, K)).astype(np.float32), rng.standard_normal((N, K) if tb else (K, N)).astype(np.float32)
    C, b = rng.standard_normal((M, N)).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    prod = (A.T if ta else A).astype(np.float64) @ (B.T if tb else B).astype(np.float64)
    for mode, tol in MODES:
        abi.nc_cuda_set_math_mode(mode)
        plain, full = torch.full((M, N), float("nan"), device="cuda"), dev(C)
        for out, alpha, beta, bias in ((plain, 1.0, 0.0, None), (full, 0.5, -2.0, b)):
            ok(abi, abi.nc_cuda_matmul_f32_ex(P(out), N, P(dev(A)), A.shape[1], P(dev(B)), B.shape[1], M, N, K, alpha, beta, ta, tb,
                                              P(dev(bias)) if bias is not None else None, None))
        close(host(plain), prod, tol)
        close(host(full), 0.5 * prod - 2.0 * C + b, tol)
