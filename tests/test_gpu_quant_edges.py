"""The activation quantiser where its shortcuts around the divisions could go wrong: quotients at and next to the middle of two
integers, scales at and next to the middle of two fp16, the ends of fp16, blocks with infinities and NaNs."""
import numpy as np
import pytest
import torch

from llamatov_b200 import _lib

pytestmark = pytest.mark.gpu


def _ulps(x, n):
    return (np.asarray(x, np.float32).view(np.int32) + np.int32(n)).view(np.float32)


def _blocks(seed):
    rng = np.random.default_rng(seed)
    out = []
    # scales around the middle of two fp16 (normal and subnormal ones, and where fp16 ends), then values around the middles of integers
    half = np.concatenate([rng.integers(1, 0x7C00, 3000), [1, 2, 3, 0x3FF, 0x400, 0x401, 0x7BFE, 0x7BFF]]).astype(np.uint16)
    lo, hi = half.view(np.float16).astype(np.float64), (half + 1).astype(np.uint16).view(np.float16).astype(np.float64)
    hi[~np.isfinite(hi)] = 65536.0
    mid = ((lo + hi) / 2 * 127).astype(np.float32)
    for k in range(-6, 7):
        amax = _ulps(mid, k)
        n = rng.integers(-127, 127, (len(amax), 31))
        with np.errstate(all="ignore"):
            d = (amax / np.float32(127)).astype(np.float16).astype(np.float32)
            v = ((n + 0.5) * d[:, None]).astype(np.float32)
        v = _ulps(v, rng.integers(-3, 4, v.shape))
        v = np.where(np.isfinite(v), v, np.float32(0))
        v = np.clip(v, -amax[:, None], amax[:, None])
        out.append(np.concatenate([amax[:, None], v], 1))
    x = np.concatenate(out)
    odd = rng.standard_normal((64, 32)).astype(np.float32) * 50
    for i, val in enumerate((np.nan, np.inf, -np.inf, 0.0, 1e-40, 3e38, -3e38)):
        odd[i::7, 5 + i] = val
    odd[3] = 0.0
    odd[10:14] *= np.float32(1e-9)
    odd[20] = np.nan
    return np.concatenate([x, odd])


def _expected(x):
    """Bytes and scales by the definition, in fp32 divisions.  The greatest value comes by a butterfly over the block, so that beside
    NaNs, which compare false, every element has its own; the block's scale is the first element's."""
    with np.errstate(all="ignore"):
        amax = np.abs(x)
        for s in (16, 8, 4, 2, 1):
            other = amax[:, np.arange(32) ^ s]
            amax = np.where(other > amax, other, amax)
        d = np.where(amax > 0, amax / np.float32(127), np.float32(1)).astype(np.float32).astype(np.float16)
        q = np.rint(x / d.astype(np.float32))
        q = np.where(np.isnan(q), 0, np.clip(q, -127, 127)).astype(np.int8)
    return q, d[:, 0].view(np.uint16)


@pytest.mark.parametrize("per_call", [8000, 1 << 20])     # a lane per value (few blocks), four values per thread
def test_quantiser_rounds_like_the_divisions(per_call):
    blocks = _blocks(1)
    assert len(blocks) > 148 * 64 * 2 and np.isnan(blocks).any(1).sum() > 8
    st = torch.cuda.current_stream().cuda_stream
    for i in range(0, len(blocks), per_call):
        b = np.ascontiguousarray(blocks[i:i + per_call])
        dx = torch.from_numpy(b).cuda()
        xq, xd = torch.empty(b.shape, dtype=torch.int8, device="cuda"), torch.empty(len(b), dtype=torch.int16, device="cuda")
        _lib.call("lt_quant_q8", dx.data_ptr(), xq.data_ptr(), xd.data_ptr(), b.size, 1, st)
        q, d = _expected(b)
        assert np.array_equal(xd.cpu().numpy().view(np.uint16), d)
        assert np.array_equal(xq.cpu().numpy(), q)


def _behind_the_norm(Wq, Wd, x, w, eps):
    """(norm, quantiser and projection one by one; the projection that does all three; the norm's output)"""
    M, K = Wq.shape
    st = torch.cuda.current_stream().cuda_stream
    n = torch.empty(K, device="cuda")
    xq, xd = torch.empty(K, dtype=torch.int8, device="cuda"), torch.empty(K // 32, dtype=torch.int16, device="cuda")
    y0, y1 = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
    _lib.call("lt_rmsnorm", x.data_ptr(), w.data_ptr(), n.data_ptr(), 1, K, eps, st)
    _lib.call("lt_quant_q8", n.data_ptr(), xq.data_ptr(), xd.data_ptr(), K, 1, st)
    _lib.call("lt_q8_gemv", Wq.data_ptr(), Wd.data_ptr(), xq.data_ptr(), xd.data_ptr(), None, y0.data_ptr(), M, K, 1, st)
    _lib.call("lt_rmsnorm_q8_gemv", Wq.data_ptr(), Wd.data_ptr(), x.data_ptr(), w.data_ptr(), eps, None, y1.data_ptr(), M, K, st)
    return y0.view(torch.int32), y1.view(torch.int32), n


def _matrix(M, K, g):
    return (torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8, device="cuda"),
            (torch.rand((M, K // 32), generator=g, device="cuda") * 0.02).half())


def test_quantiser_behind_the_norm_rounds_like_the_separate_one():
    """The projection that normalises and quantises for itself against norm, quantiser and projection: the same bits, also for
    rows with a NaN or an infinity, whose norm every value sees."""
    K, g = 1152, torch.Generator(device="cuda").manual_seed(4)
    Wq, Wd = _matrix(64, K, g)
    w = torch.randn(K, generator=g, device="cuda")
    for scale, odd in ((1.0, 0.0), (1e-12, 0.0), (3e4, 0.0), (1.0, float("nan")), (1.0, float("inf"))):
        x = torch.randn(K, generator=g, device="cuda") * scale
        if odd:
            x[77] = odd
        y0, y1, _ = _behind_the_norm(Wq, Wd, x, w, 1e-5)
        assert torch.equal(y0, y1)
    assert _lib.device_status() == set()


def test_quantiser_behind_the_norm_at_the_boundaries():
    """The same where the norm's output is its weight (rows of ones, no epsilon): the blocks above, whose values lie at the middles of
    integers and whose scales at the middles of fp16, 36 a call."""
    K, g = 1152, torch.Generator(device="cuda").manual_seed(5)
    Wq, Wd = _matrix(64, K, g)
    blocks = _blocks(2)
    blocks = blocks[np.isfinite(blocks).all(1)]
    x = torch.ones(K, device="cuda")
    for i in range(0, len(blocks) - 36, len(blocks) // 300):
        w = torch.from_numpy(blocks[i:i + 36].reshape(-1)).cuda()
        y0, y1, n = _behind_the_norm(Wq, Wd, x, w, 0.0)
        assert torch.equal(n, w) and torch.equal(y0, y1)
    assert _lib.device_status() == set()
