"""Row maxima of prompt attention from 16-bit products: the bits of the exact search whatever the scores are."""
import pytest
import torch

from llamatov_b200 import _lib

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def attend(Q, K, V, T, L, hd, nh, nkv, scale):
    out, ln = torch.full((T, nh * hd), 7.0, device="cuda"), torch.tensor([L], dtype=torch.int32, device="cuda")
    _lib.call("lt_attn_prefill", Q.data_ptr(), nh * hd, K.data_ptr(), V.data_ptr(), ln.data_ptr(), out.data_ptr(), nh * hd, hd, nh, nkv, scale, T, L,
              torch.cuda.current_stream().cuda_stream)
    return out


# spread scores; one greatest for all rows; all equal; closer than 16 bits tell apart; whole numbers (ties); not finite in a key or a
# query; beyond what a squared norm holds; below it
EDITS = {
    "plain": lambda q, k: None, "one": lambda q, k: k[1].mul_(50), "equal": lambda q, k: k.copy_(k[:1].expand_as(k)),
    "near": lambda q, k: k.copy_(k[:1] + 1e-4 * k), "ties": lambda q, k: (q.round_(), k.round_()), "zero": lambda q, k: q.zero_(),
    "inf": lambda q, k: k[7].fill_(INF), "nan": lambda q, k: k[9, ::5].fill_(NAN), "nan-q": lambda q, k: q[3, 5].fill_(NAN),
    "big": lambda q, k: (q.mul_(1e14), k.mul_(1e14)), "over": lambda q, k: (q.mul_(1e25), k.mul_(1e25)),
    "small": lambda q, k: (q.mul_(1e-22), k.mul_(1e-22)), "subnormal": lambda q, k: (q.mul_(1e-39), k.mul_(1e18))}


@pytest.mark.parametrize("name", EDITS)
@pytest.mark.parametrize("hd,nh,nkv,T,L0,scale", [(64, 14, 2, 1025, 3, 0.125), (128, 32, 8, 450, 64, 128 ** -0.5), (64, 30, 2, 515, 5, -0.3)])
def test_row_maxima_bit_exact(name, hd, nh, nkv, T, L0, scale):
    g = torch.Generator(device="cuda").manual_seed(T)
    L = L0 + T
    Q, K, V = (torch.randn((n, w * hd), device="cuda", generator=g) for n, w in ((T, nh), (L, nkv), (L, nkv)))
    EDITS[name](Q, K)
    got = attend(Q, K, V, T, L, hd, nh, nkv, scale)
    for r in range(0, T, 31):               # the same rows in chunks that take the form without tiles of 32 rows
        n = min(31, T - r)
        want = attend(Q[r:], K, V, n, L0 + r + n, hd, nh, nkv, scale)
        assert torch.equal(got[r:r + n].nan_to_num(nan=123.0), want.nan_to_num(nan=123.0)), (name, r)
    assert _lib.device_status() == set()


# One large element that q and all keys share, as projections with a bias produce: it takes the rounding error of 16 bits to one side in
# every key.  Its value is just below the middle of two neighbours with `bits` significant ones, the keys' spread below it.
def _shared(bits, spread, noise, big=8.0):
    def edit(q, k, g):
        q.mul_(noise)
        k.mul_(noise)
        q[..., 0] = big * (1 + 0.98 * 2.0 ** -bits)
        k[..., 0] = big * (1 + 0.98 * 2.0 ** -bits) * (1 - spread * torch.rand(k.shape[:2], device="cuda", generator=g))
    return edit


def _two_keys(bits):      # the greatest score loses most by rounding, the next one nothing
    def edit(q, k, g):
        q.zero_()
        k.zero_()
        q[..., 0] = 1 + 0.98 * 2.0 ** -bits
        k[3, :, 0] = 1 + 0.98 * 2.0 ** -bits
        k[7, :, 0], k[7, :, 1] = 1 + 0.8 * 2.0 ** -bits, 1
    return edit


SIXTEEN = {f"shared-{b}-{s}-{n}": _shared(b, s, n) for b in (8, 11) for s in (2.0 ** -b, 2.0 ** (2 - b), 0.01) for n in (0, 0.05)}
SIXTEEN |= {f"biased-{b}": _shared(b, 0.002, 1.0, 100.0) for b in (8, 11)} | {f"two-{b}": _two_keys(b) for b in (8, 11)}
# about half of the elements below the normal fp16; norms just inside and just beyond what fp16 may hold
TIMES = {"small": (1e-3, 1e-4), "inside": (6e3, 6e3), "beyond": (1e4, 1e4)}
SIXTEEN |= {n: lambda q, k, g, t=t: (q.mul_(t[0]), k.mul_(t[1])) for n, t in TIMES.items()}


@pytest.mark.parametrize("name", SIXTEEN)
@pytest.mark.parametrize("hd,nh,nkv,T,L0", [(64, 14, 2, 1025, 3), (128, 32, 8, 450, 64)])
def test_row_maxima_where_sixteen_bits_round_to_one_side(name, hd, nh, nkv, T, L0):
    g = torch.Generator(device="cuda").manual_seed(T)
    L = L0 + T
    Q, K, V = (torch.randn((n, w, hd), device="cuda", generator=g) for n, w in ((T, nh), (L, nkv), (L, nkv)))
    a, b = TIMES.get(name, (1.0, 1.0))
    scale = hd ** -0.5 / (a * b)            # scores of ordinary size
    SIXTEEN[name](Q, K, g)
    Q, K = Q.reshape(T, -1), K.reshape(L, -1)
    got = attend(Q, K, V, T, L, hd, nh, nkv, scale)
    for r in range(0, T, 31):
        n = min(31, T - r)
        want = attend(Q[r:], K, V, n, L0 + r + n, hd, nh, nkv, scale)
        assert torch.equal(got[r:r + n], want), (name, r)
    assert torch.isfinite(got).all() and _lib.device_status() == set()


@pytest.mark.parametrize("hd,nh,nkv,T,L0", [(64, 14, 2, 700, 3), (128, 16, 4, 832, 0), (64, 14, 2, 333, 0), (64, 14, 2, 20, 9)])
def test_rows_whose_scores_are_all_below_the_mask(hd, nh, nkv, T, L0):
    """Scores of minus infinity, and below -1e30, throughout a row: zeros, as from the one-token kernel, in every form (32 rows per
    CTA, 16, fewer) and wherever in its tile the row is."""
    g = torch.Generator(device="cuda").manual_seed(T)
    L = L0 + T
    Q, K, V = (torch.randn((n, w, hd), device="cuda", generator=g) for n, w in ((T, nh), (L, nkv), (L, nkv)))
    K[..., 0] = 1 + K[..., 0].abs()
    rows = [r for r in (0, 5, 7, 15, 16, 31, 33, T - 1) if r < T]
    for i, r in enumerate(rows):
        Q[r] = 0
        Q[r, :, 0] = (-INF, -1e38)[i % 2]
    Q, K = Q.reshape(T, -1), K.reshape(L, -1)
    got = attend(Q, K, V, T, L, hd, nh, nkv, 0.125)
    assert (got[rows] == 0).all() and torch.isfinite(got).all()
    one, Kr, Vr = torch.empty(nh * hd, device="cuda"), torch.cat([K, K[:1]]), torch.cat([V, V[:1]])      # room for one more position
    for r in rows + [T // 2]:
        ln = torch.tensor([L0 + r + 1], dtype=torch.int32, device="cuda")
        _lib.call("lt_attn_decode_masked", Q[r].data_ptr(), Kr.data_ptr(), Vr.data_ptr(), ln.data_ptr(), one.data_ptr(), hd, nh, nkv, 0.125, L + 1,
                  torch.cuda.current_stream().cuda_stream)
        assert torch.equal(one, got[r]), r
    assert _lib.device_status() == set()
