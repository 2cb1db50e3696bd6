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
    """Bytes and scales by the definition, in fp32 divisions; None for blocks with NaNs."""
    with np.errstate(all="ignore"):
        amax = np.abs(x).max(1)
        d = np.where(amax > 0, amax / np.float32(127), np.float32(1)).astype(np.float32).astype(np.float16)
        q = np.rint(x / d.astype(np.float32)[:, None])
        q = np.where(np.isnan(q), 0, np.clip(q, -127, 127)).astype(np.int8)
    return q, d.view(np.uint16)


@pytest.mark.parametrize("rows", [1, 40])     # a lane per value, four values per thread
def test_quantiser_rounds_like_the_divisions(rows):
    x = _blocks(rows)
    x = x[:len(x) // rows * rows].reshape(rows, -1) if rows > 1 else x.reshape(1, -1)
    if rows == 1:
        x = x[:, :32 * 2000]                  # few blocks: the form with a lane per value
        x[:, -32 * 64:] = _blocks(1)[-64:].reshape(1, -1)
    K = x.shape[1]
    dx = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    xq, xd = torch.empty(x.shape, dtype=torch.int8, device="cuda"), torch.empty((rows, K // 32), dtype=torch.int16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.call("lt_quant_q8", dx.data_ptr(), xq.data_ptr(), xd.data_ptr(), K, rows, st)
    b = x.reshape(-1, 32)
    q, d = _expected(b)
    ok = ~np.isnan(b).any(1)
    assert ok.sum() > 1000
    assert np.array_equal(xd.cpu().numpy().view(np.uint16).reshape(-1)[ok], d[ok])
    assert np.array_equal(xq.cpu().numpy().reshape(-1, 32)[ok], q[ok])


def test_quantiser_behind_the_norm_rounds_like_the_separate_one():
    """The projection that normalises and quantises for itself against norm, quantiser and projection: the same bits, NaNs
    (which every value of a row sees) included."""
    K, M, st = 1152, 64, torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(4)
    Wq = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8, device="cuda")
    Wd = (torch.rand((M, K // 32), generator=g, device="cuda") * 0.02).half()
    w = torch.randn(K, generator=g, device="cuda")
    for scale in (1.0, 1e-12, 3e4):
        x = torch.randn(K, generator=g, device="cuda") * scale
        n = torch.empty(K, device="cuda")
        xq, xd = torch.empty(K, dtype=torch.int8, device="cuda"), torch.empty(K // 32, dtype=torch.int16, device="cuda")
        y0, y1 = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
        _lib.call("lt_rmsnorm", x.data_ptr(), w.data_ptr(), n.data_ptr(), 1, K, 1e-5, st)
        _lib.call("lt_quant_q8", n.data_ptr(), xq.data_ptr(), xd.data_ptr(), K, 1, st)
        _lib.call("lt_q8_gemv", Wq.data_ptr(), Wd.data_ptr(), xq.data_ptr(), xd.data_ptr(), None, y0.data_ptr(), M, K, 1, st)
        _lib.call("lt_rmsnorm_q8_gemv", Wq.data_ptr(), Wd.data_ptr(), x.data_ptr(), w.data_ptr(), 1e-5, None, y1.data_ptr(), M, K, st)
        assert torch.equal(y0.view(torch.int32), y1.view(torch.int32))
    assert _lib.device_status() == set()
