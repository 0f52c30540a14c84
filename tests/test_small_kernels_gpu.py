"""The CUDA-core kernels for small problems against the float64 oracle, at the edges of their tiles: one and a few rows, sums
shorter than a warp, sizes that are no multiple of four (scalar accesses) or of a tile, more blocks than one reduction group."""
import numpy as np
import pytest

from oracle import nocta_oracle as O
from tests.test_abi_gpu import MODE_SIMT, MODE_TF32, P, TOL_F32, _release_uploads, abi, close, dev, host, ok  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _plain_f32_outputs(abi):  # noqa: F811
    abi.nc_cuda_set_round_outputs(0)   # whatever ran before in this process: results are compared as plain f32


# rows, inputs, outputs: below and at the row tiles (1, 2, 4, 8, 16), several row tiles, k not a multiple of 4 / 32 / 128,
# one output, ten outputs over a long sum, the largest product that stays on these kernels
LINEAR = [(1, 84, 10), (2, 31, 5), (3, 130, 17), (5, 256, 120), (8, 1, 3), (16, 1024, 260), (17, 515, 33), (64, 256, 120), (31, 7, 1),
          (128, 8192, 10), (100, 37, 129), (127, 250, 501)]


@pytest.mark.parametrize("mode", [MODE_SIMT, MODE_TF32])
@pytest.mark.parametrize("B,I,Oo", LINEAR)
def test_small_linear(abi, mode, B, I, Oo):  # noqa: F811
    rng = np.random.default_rng(B * 131 + I * 7 + Oo)
    x, W = rng.standard_normal((B, I)).astype(np.float32), (rng.standard_normal((Oo, I)) / np.sqrt(I)).astype(np.float32)
    b, g = rng.standard_normal(Oo).astype(np.float32), rng.standard_normal((B, Oo)).astype(np.float32)
    abi.nc_cuda_set_math_mode(mode)
    nan = lambda *s: torch.full(s, float("nan"), device="cuda")  # noqa: E731
    y, gx, gW, gb = nan(B, Oo), nan(B, I), nan(Oo, I), nan(Oo)
    tx, tW, tg = dev(x), dev(W), dev(g)
    ok(abi, abi.nc_cuda_linear_forward_f32_ex(P(y), P(tx), P(tW), P(dev(b)), B, I, Oo, None))
    ok(abi, abi.nc_cuda_linear_backward_f32_ex(P(gx), P(gW), P(gb), P(tg), P(tx), P(tW), B, I, Oo, None))
    # TF32 mode reads the weights of 128 and more rows rounded to TF32 (off by up to 2^-11); against those the sums are f32 again
    Wr = W if mode == MODE_SIMT or B < 128 else ((W.view(np.uint32) + np.uint32(0x1000)) & np.uint32(0xFFFFE000)).view(np.float32)
    dx, dW, db = O.linear_backward(g, x, Wr)
    close(host(y), O.linear_forward(x, Wr, b), TOL_F32)
    close(host(gx), dx, TOL_F32)
    close(host(gW), dW, TOL_F32)
    close(host(gb), db, TOL_F32)


# N, Cin, H, W, Cout, k, pad: widths around the four-pixel groups, channels around the four-channel groups, sliced and unsliced input
# channels, one image and more images than SMs (several per block), all filter sizes, outputs smaller than one group
CONV = [(1, 1, 28, 28, 6, 5, 0), (1, 6, 12, 12, 16, 5, 0), (3, 2, 7, 9, 3, 3, 1), (2, 5, 5, 5, 1, 5, 0), (2, 3, 9, 6, 4, 7, 3), (170, 1, 10, 11, 6, 5, 0),
        (301, 6, 12, 12, 16, 5, 0), (2, 15, 8, 13, 32, 3, 0), (2, 32, 8, 13, 15, 3, 1), (9, 4, 33, 3, 5, 3, 1), (2, 8, 6, 6, 8, 3, 2)]


@pytest.mark.parametrize("N,Ci,H,W,Co,k,p", CONV)
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
def test_small_conv(abi, layout, N, Ci, H, W, Co, k, p):  # noqa: F811
    from nocta_b200.cuda_abi import size4
    rng = np.random.default_rng(N + 3 * Ci + 5 * H + 7 * W + Co + k)
    x, w = rng.standard_normal((N, Ci, H, W)).astype(np.float32), (rng.standard_normal((Co, Ci, k, k)) / np.sqrt(Ci * k * k)).astype(np.float32)
    b = rng.standard_normal(Co).astype(np.float32)
    yo = O.conv2d_forward(x, w, b, 1, p)
    Ho, Wo = yo.shape[2:]
    g = rng.standard_normal(yo.shape).astype(np.float32)
    dxo, dwo, dbo = O.conv2d_backward(x, w, g, 1, p)
    abi.nc_cuda_set_math_mode(MODE_TF32)
    cl = layout == "nhwc"
    put = lambda a: dev(a.transpose(0, 2, 3, 1) if cl else a)  # noqa: E731
    get = lambda t, shape: host(t).reshape(shape[0], shape[2], shape[3], shape[1]).transpose(0, 3, 1, 2) if cl else host(t).reshape(shape)  # noqa: E731
    strides = lambda C, h, v: size4([h * v * C, 1, v * C, C] if cl else [C * h * v, h * v, v, 1])  # noqa: E731
    xs, ys = strides(Ci, H, W), strides(Co, Ho, Wo)
    nan = lambda n: torch.full((n,), float("nan"), device="cuda")  # noqa: E731
    y, gx, gw, gb = nan(yo.size), nan(x.size), nan(w.size), nan(Co)
    tx, tg, tw = put(x), put(g), dev(w)
    for _ in range(2):   # twice: the weight gradient's arrival counter has to come back to zero by itself
        ok(abi, abi.nc_cuda_conv2d_forward_f32_ex(P(y), ys, P(tx), xs, P(tw), P(dev(b)), N, Ci, H, W, Co, k, k, 1, p, None))
        ok(abi, abi.nc_cuda_conv2d_backward_weight_f32_ex(P(gw), P(gb), P(tg), ys, P(tx), xs, N, Ci, H, W, Co, k, k, 1, p, None))
        ok(abi, abi.nc_cuda_conv2d_backward_input_f32_ex(P(gx), xs, P(tg), ys, P(tw), N, Ci, H, W, Co, k, k, 1, p, None))
        close(get(y, yo.shape), yo, TOL_F32)
        close(get(gx, x.shape), dxo, TOL_F32)
        close(host(gw).reshape(w.shape), dwo, TOL_F32)
        close(host(gb), dbo, TOL_F32)


def test_small_conv_infinity(abi):  # noqa: F811
    """An infinity in the last input column reaches the weight gradient's last filter column only, also beside the padding of a row
    group of four (seven output columns)."""
    from nocta_b200.cuda_abi import size4
    H = W = 9
    x, g = np.ones((1, 1, H, W), np.float32), np.ones((1, 2, 7, 7), np.float32)
    x[0, 0, 0, 8] = np.inf
    abi.nc_cuda_set_math_mode(MODE_TF32)
    gw = torch.zeros(18, device="cuda")
    ok(abi, abi.nc_cuda_conv2d_backward_weight_f32_ex(P(gw), None, P(dev(g)), size4([98, 49, 7, 1]), P(dev(x)), size4([81, 81, 9, 1]),
                                                      1, 1, H, W, 2, 3, 3, 1, 0, None))
    got = host(gw).reshape(2, 3, 3)
    assert np.isposinf(got[:, 0, 2]).all()
    got[:, 0, 2] = 49.0
    assert (got == 49.0).all()


# rows x columns: a row per block and a row per warp (2368 rows and more), vector and scalar columns, the most columns a block's
# registers hold, and more than that
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 31), (16, 1024), (2, 8192), (2, 8196), (5, 1025), (2400, 64), (2400, 310), (2500, 1024), (2500, 1028)])
def test_layernorm_rows(abi, rows, cols):  # noqa: F811
    rng = np.random.default_rng(rows + cols)
    x, g = rng.standard_normal((rows, cols)).astype(np.float32) + 1.5, rng.standard_normal((rows, cols)).astype(np.float32)
    ga, be = rng.standard_normal(cols).astype(np.float32), rng.standard_normal(cols).astype(np.float32)
    y, gx, dga, dbe = (torch.full(s, float("nan"), device="cuda") for s in ((rows, cols), (rows, cols), (cols,), (cols,)))
    tx, tga = dev(x), dev(ga)
    ok(abi, abi.nc_cuda_layernorm_forward_f32_ex(P(y), P(tx), P(tga), P(dev(be)), rows, cols, 1e-5, None))
    ok(abi, abi.nc_cuda_layernorm_backward_f32_ex(P(gx), P(dga), P(dbe), P(dev(g)), P(tx), P(tga), rows, cols, 1e-5, None))
    x64, g64 = x.astype(np.float64), g.astype(np.float64)
    mu, var = x64.mean(1, keepdims=True), x64.var(1, keepdims=True)
    xh = (x64 - mu) / np.sqrt(var + 1e-5)
    gg = g64 * ga
    dx = (gg - gg.mean(1, keepdims=True) - xh * (gg * xh).mean(1, keepdims=True)) / np.sqrt(var + 1e-5)
    close(host(y), xh * ga + be, TOL_F32)
    if cols > 1:   # a row of one value has a zero gradient
        close(host(gx), dx, TOL_F32)
    close(host(dga), (g64 * xh).sum(0), TOL_F32)
    close(host(dbe), g64.sum(0), TOL_F32)


@pytest.mark.parametrize("n", [1, 5, 4096, 1000003])
def test_mse_sizes(abi, n):  # noqa: F811
    rng = np.random.default_rng(n)
    p, t = rng.standard_normal(n).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    for off in (0, 1):   # aligned and unaligned operands
        tp, tt = dev(np.concatenate([np.zeros(off, np.float32), p]))[off:], dev(np.concatenate([np.zeros(off, np.float32), t]))[off:]
        loss, gp = torch.full((1,), float("nan"), device="cuda"), torch.full((n,), float("nan"), device="cuda")
        ok(abi, abi.nc_cuda_mse_fused_f32_ex(P(loss), P(gp), None, P(tp), P(tt), n, 1.0, None))
        d = p.astype(np.float64) - t
        close(host(loss), np.array([(d * d).mean()]), TOL_F32)
        close(host(gp), 2.0 * d / n, TOL_F32)


# first layer (3 input channels): channel counts that fill 32, 64 or 128 padded channels only in part, more than one group of 64, more
# than the tiled forward kernel takes; image widths around the 64-pixel strip
@pytest.mark.parametrize("N,H,W,Co", [(2, 9, 70, 48), (3, 5, 64, 16), (1, 12, 13, 80), (2, 7, 65, 112), (2, 6, 6, 176), (5, 10, 3, 96)])
def test_first_layer_channels(abi, N, H, W, Co):  # noqa: F811
    from nocta_b200.cuda_abi import size4
    rng = np.random.default_rng(N + H + W + Co)
    x, w, b = (rng.standard_normal(s).astype(np.float32) for s in ((N, 3, H, W), (Co, 3, 3, 3), (Co,)))
    g = rng.standard_normal((N, Co, H, W)).astype(np.float32)
    _, dwo, dbo = O.conv2d_backward(x, w, g, 1, 1)
    abi.nc_cuda_set_math_mode(MODE_TF32)
    xs, ys = size4([3 * H * W, H * W, W, 1]), size4([H * W * Co, 1, W * Co, Co])
    nan = lambda n: torch.full((n,), float("nan"), device="cuda")  # noqa: E731
    y, gw, gb, tx, tg = nan(g.size), nan(w.size), nan(Co), dev(x), dev(g.transpose(0, 2, 3, 1))
    ok(abi, abi.nc_cuda_conv2d_forward_f32_ex(P(y), ys, P(tx), xs, P(dev(w)), P(dev(b)), N, 3, H, W, Co, 3, 3, 1, 1, None))
    ok(abi, abi.nc_cuda_conv2d_backward_weight_f32_ex(P(gw), P(gb), P(tg), ys, P(tx), xs, N, 3, H, W, Co, 3, 3, 1, 1, None))
    close(host(y).reshape(N, H, W, Co).transpose(0, 3, 1, 2), O.conv2d_forward(x, w, b, 1, 1), TOL_F32)
    close(host(gw).reshape(w.shape), dwo, TOL_F32)
    close(host(gb), dbo, TOL_F32)
