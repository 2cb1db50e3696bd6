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
