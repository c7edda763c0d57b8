"""GPU check of the tensor-core convolutions' tiles on small and ragged grids: lines of one
voxel to more than two tiles, tiles that end on, before and after a line, every number of
input channel chunks, and output widths on both sides of the weight gradient's split of
the taps.  The reference is the sum over the taps in float64 on the same BF16 values."""
import numpy as np
import pytest

import saras_gb300 as S

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (5, 4, 1), (1, 2, 126), (2, 1, 127), (3, 2, 128), (2, 3, 63), (1, 1, 300), (4, 5, 9)]
CHANNELS = [(16, 16), (48, 32), (64, 16), (96, 96), (16, 96)]


def taps(x, D, H, W):
    p = np.zeros((D + 2, H + 2, W + 2, x.shape[-1]))
    p[1:-1, 1:-1, 1:-1] = x
    return [p[z:z + D, y:y + H, k:k + W] for z in range(3) for y in range(3) for k in range(3)]


def check(got, ref, size, terms):
    """got is the BF16 rounding of a value within terms 2^-24 size of ref (rounding is monotone)."""
    tol = terms * 2.0 ** -24 * size + 1e-30
    lo, hi = (S.from_bf16_bits(S.to_bf16_bits((ref + q).astype(np.float32))) for q in (-tol, tol))
    g = got.reshape(ref.shape)
    assert np.all((g >= lo) & (g <= hi)), float(np.max(np.abs(g - ref)))


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("cin,cout", CHANNELS)
def test_conv_tiles(dims, cin, cout):
    """BF16 results: the rounding of a value that FP32 sums of 27 cin terms can give (2^-24 a
    term of the terms' absolute sum).  FP32 weight gradients: 2^-23 a term."""
    D, H, W = dims
    rng = np.random.default_rng(5)
    xb = S.to_bf16_bits(rng.standard_normal((D, H, W, cin)).astype(np.float32))
    db = S.to_bf16_bits(rng.standard_normal((D, H, W, cout)).astype(np.float32))
    w = S.from_bf16_bits(S.to_bf16_bits((rng.standard_normal((cout, 27, cin)) / np.sqrt(27 * cin)).astype(np.float32)))
    b = rng.standard_normal(cout).astype(np.float32)
    x, dy, w64 = (S.from_bf16_bits(q).astype(np.float64) for q in (xb, db, S.to_bf16_bits(w)))
    x, dy, w64 = x.reshape(D, H, W, cin), dy.reshape(D, H, W, cout), w64.reshape(cout, 27, cin)

    ref = b + sum(t @ w64[:, q].T for q, t in enumerate(taps(x, D, H, W)))
    size = np.abs(b) + sum(t @ np.abs(w64[:, q]).T for q, t in enumerate(taps(np.abs(x), D, H, W)))
    check(S.conv3d_check(0, xb, None, w, b, 0, dims, cin, cout), ref, size, 27 * cin + 1)
    ref = sum(t @ w64[:, 26 - q] for q, t in enumerate(taps(dy, D, H, W)))
    size = sum(t @ np.abs(w64[:, 26 - q]) for q, t in enumerate(taps(np.abs(dy), D, H, W)))
    check(S.conv3d_check(1, None, db, w, None, 0, dims, cin, cout), ref, size, 27 * cout)
    got = S.conv3d_check(2, xb, db, w, None, 0, dims, cin, cout)
    ref = np.stack([np.einsum("zyxn,zyxc->nc", dy, t) for t in taps(x, D, H, W)], 1)
    size = np.stack([np.einsum("zyxn,zyxc->nc", np.abs(dy), t) for t in taps(np.abs(x), D, H, W)], 1)
    err = np.abs(got[:27 * cin * cout].reshape(cout, 27, cin) - ref)
    n = D * H * W
    assert np.all(err <= n * 2.0 ** -23 * size), float(np.max(err))
    assert np.all(np.abs(got[27 * cin * cout:] - dy.reshape(n, cout).sum(0)) <= n * 2.0 ** -23 * np.abs(dy).reshape(n, cout).sum(0))


def test_conv_tiles_five_chunks():
    """80 input channels (rows dealt to 120 threads), forward."""
    D, H, W, cin, cout = 2, 3, 70, 80, 32
    rng = np.random.default_rng(6)
    xb = S.to_bf16_bits(rng.standard_normal((D, H, W, cin)).astype(np.float32))
    w = S.from_bf16_bits(S.to_bf16_bits((rng.standard_normal((cout, 27, cin)) / np.sqrt(27 * cin)).astype(np.float32)))
    x = S.from_bf16_bits(xb).astype(np.float64).reshape(D, H, W, cin)
    w64 = w.astype(np.float64).reshape(cout, 27, cin)
    ref = sum(t @ w64[:, q].T for q, t in enumerate(taps(x, D, H, W)))
    size = sum(t @ np.abs(w64[:, q]).T for q, t in enumerate(taps(np.abs(x), D, H, W)))
    check(S.conv3d_check(0, xb, None, w, None, 0, (D, H, W), cin, cout), ref, size, 27 * cin)
