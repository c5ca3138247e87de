"""Register-tiled sweeps of the backward against the oracle at the edges of their tiles: lengths around
a block of 16 rows and a band of 256 diagonals, symbols on both sides of 8 bits (the row sums' tile
holds 8 or 16), all value widths, launches of little and of much work (one, two or four diagonals per
thread), and streams whose window products stay alive (S rebuilt from every fourth row together with
the products)."""
import hashlib

import numpy as np
import pytest
import torch

from tests.helpers import grad_tol, nonzero_randn, normalised_error, oracle_grads, repeated_stream_logits

pytestmark = pytest.mark.gpu
DEV = "cuda"

DTYPES = (torch.float32, torch.float16, torch.bfloat16)


def _check(q, k, v, go, shape, W, p, m, dtype):
    from rosa_soft_b200 import cabi
    B, T = shape
    q, k, v, go = (t.to(dtype).to(DEV) for t in (q, k, v, go))
    cu = np.arange(B + 1, dtype=np.int64) * T
    _, pq, pk, _, _ = cabi.hard_forward(q, k, v, shape, W)
    seed = torch.tensor(7, dtype=torch.int64, device=DEV) if p > 0 else None
    got = cabi.surrogate_vjp(q, k, v, go, shape, pq, pk, W, 1.0, p, m, seed, 7)[:3]
    want = oracle_grads(q, k, v, go, cu, W, 1.0, p, m, 7)
    # the bounds of the operand terms that the contraction keeps (tests/helpers.py)
    for mine, ref in zip(got, want):
        assert normalised_error(mine.cpu().numpy(), ref) <= grad_tol(dtype)


def _random(B, T, H, D, Hv, Dv, W, p, dtype):
    q, k = (nonzero_randn((B * T, H, D), T + s) for s in (1, 2))
    _check(q, k, nonzero_randn((B * T, Hv, Dv), T + 3), nonzero_randn((B * T, H, Dv), T + 4), (B, T), W, p, 3.0,
           dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,D,Dv,W,p", [
    (15, 7, 5, 4, 0.0), (17, 8, 8, 40, 0.1), (256, 8, 16, 3, 0.0), (257, 9, 16, 30, 0.1), (273, 16, 13, 30, 0.0),
    (530, 8, 8, 128, 0.1), (514, 9, 32, 60, 0.05), (289, 8, 24, 17, 0.0), (600, 1, 4, 9, 0.1)])
def test_tile_edges(T, D, Dv, W, p, dtype):
    _random(2, T, 2, D, 1, Dv, W, p, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,D,Dv,W,p", [
    (600, 2, 8, 20, 0.0), (700, 1, 16, 1, 0.1), (530, 8, 8, 2, 0.0), (540, 3, 32, 33, 0.1), (520, 10, 6, 15, 0.0)])
def test_live_window_products(T, D, Dv, W, p, dtype):
    H = 2
    q = repeated_stream_logits(T, H, D, seed=T)
    _check(q, q.clone(), nonzero_randn((T, H, Dv), 3), nonzero_randn((T, H, Dv), 4), (1, T), W, p, 3.0, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("B,H,T,D,Dv,W,p", [
    (1, 2, 257, 17, 8, 40, 0.1), (1, 2, 531, 24, 32, 30, 0.05), (1, 1, 290, 32, 15, 300, 0.1),     # one diagonal
    (9, 32, 261, 8, 8, 20, 0.1), (9, 32, 258, 4, 16, 300, 0.0), (9, 32, 257, 20, 24, 20, 0.1),     # two
    (33, 32, 129, 6, 12, 20, 0.1), (33, 32, 146, 8, 4, 200, 0.1), (33, 32, 100, 9, 20, 7, 0.05)])  # four, four, two
def test_launches_of_every_size(B, H, T, D, Dv, W, p, dtype):
    _random(B, T, H, D, 1, Dv, W, p, dtype)


# sha256 of the float32 gradients (dq, dk, dv) of heads 0 and 1 of sequence 0, as the sweep with four
# diagonals per thread gave them before there were others.  No window product is alive here.
ROW_SUM_BITS = {
    (8, 0.0): "06e1d9c03c593cb661cc5a2ffafa681bbd012a46286ddcd7a991cb0187fd1e16",
    (8, 0.1): "4245b35eeb36ebe843df237814b20e7384b4a9d709be7167e5379488741a90e1",
    (16, 0.1): "9d38878ae149926d4f5f5513b906890efed4f8822f673d9ef63a730a2ec79c05",
    (24, 0.0): "c474b1a2f15a05974865e01d01a14666bcaa9df7901daee8027ab75b6ca4a24f"}


@pytest.mark.parametrize("B,H", [(1, 4), (1, 256), (32, 64)])       # one, two, four diagonals per thread
@pytest.mark.parametrize("Dv,p", sorted(ROW_SUM_BITS))
def test_row_sums_have_the_same_bits_in_launches_of_every_size(B, H, Dv, p):
    from rosa_soft_b200 import cabi
    T, D, W = 530, 8, 128
    whole = lambda x: x.repeat(B, H // 2, 1).to(DEV)  # noqa: E731
    q, k, v, go = (whole(nonzero_randn((T, 2, n), s)) for s, n in ((1, D), (2, D), (3, Dv), (4, Dv)))
    _, pq, pk, _, _ = cabi.hard_forward(q, k, v, (B, T), W)
    seed = torch.tensor(7, dtype=torch.int64, device=DEV) if p > 0 else None
    got = cabi.surrogate_vjp(q, k, v, go, (B, T), pq, pk, W, 1.0, p, 3.0, seed, 7)[:3]
    bits = hashlib.sha256(b"".join(g[:T, :2].contiguous().cpu().numpy().tobytes() for g in got)).hexdigest()
    assert bits == ROW_SUM_BITS[Dv, p]


@pytest.mark.parametrize("W,m", [(2, 3.0), (3, 9.0), (5, 6.0), (16, 3.0)])
def test_runs_of_matches_far_longer_than_the_horizon(W, m):
    """Lone mismatches between long runs: products on both sides of the cut-off, and an adjoint that adds up
    over a whole run."""
    T, H, D = 1200, 2, 2
    rng = np.random.default_rng(W)
    tokens = np.repeat(rng.integers(0, 4, size=(T // 8, H)), 8, axis=0)
    tokens[rng.integers(0, T, size=40), 0] ^= 3
    q = torch.from_numpy(np.where((tokens[..., None] >> np.arange(D)) & 1, 0.7, -0.7).astype(np.float32))
    _check(q, q.clone(), nonzero_randn((T, H, 8), 3), nonzero_randn((T, H, 8), 4), (1, T), W, 0.0, m,
           torch.float32)
