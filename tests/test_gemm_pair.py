"""The Q8_0 GEMM with 32-column tiles (form 6 of lt_q8_gemm_tc): its bits, and where the default takes it."""
import numpy as np
import pytest
import torch

from llamatov_b200 import _lib, synth


# us on a B200 (148 SMs; 72 and 33 clusters at once): the 16-column tiles as the default splits them, form 6
MEASURED = [
    ((128, 512, 2048), (6.0, 8.7)), ((896, 896, 64), (6.7, 9.3)), ((896, 896, 1000), (15.5, 14.7)), ((896, 896, 2048), (31.0, 22.0)),
    ((1152, 896, 2048), (36.7, 24.0)), ((9728, 896, 16), (7.4, 10.6)), ((9728, 896, 333), (50.0, 32.3)), ((9728, 896, 2048), (264.1, 140.3)),
    ((896, 4864, 64), (13.0, 24.7)), ((896, 4864, 2048), (111.6, 77.0)), ((2048, 4096, 96), (17.2, 20.3)), ((4096, 4096, 32), (14.5, 21.6)),
    ((4096, 4096, 64), (18.2, 21.5)), ((4096, 4096, 128), (32.2, 21.9)), ((6144, 4096, 32), (18.2, 21.8)), ((6144, 4096, 64), (32.7, 22.0)),
    ((28672, 4096, 16), (36.6, 42.4)), ((28672, 4096, 32), (61.5, 44.6)), ((28672, 4096, 512), (683.1, 379.0)),
    ((4096, 14336, 32), (36.0, 64.6)), ((4096, 14336, 128), (100.6, 62.9)),
]


@pytest.mark.parametrize("size,us", MEASURED)
def test_the_default_is_the_faster_form(size, us):
    """The choice is host arithmetic over two fitted costs: this holds its constants to times measured apart from it (it times
    nothing itself).  6 % is what a shape near the line may lose."""
    pair = _lib.lib().lt_q8_gemm_tc_pair(*size, 148, 72, 33)
    assert us[pair] <= 1.06 * min(us)


def test_what_the_default_refuses_stays_with_it():
    pair = _lib.lib().lt_q8_gemm_tc_pair
    assert pair(4096, 1 << 17, 512, 148, 72, 33) == 0       # rows whose scales the 16-column tiles cannot hold: refused, not taken
    assert pair(896, 4864 + 32, 512, 148, 72, 33) == 0 and pair(0, 4864, 512, 148, 72, 33) == 0


def _gemm(Wq, Wd, Xq, Xd, M, K, T, variant, resid=None, ld=0):
    y = torch.full((T, M), float("nan"), device="cuda")
    _lib.call("lt_q8_gemm_tc", Wq.data_ptr(), Wd.data_ptr(), Xq.data_ptr(), Xd.data_ptr(), None if resid is None else resid.data_ptr(), ld,
              y.data_ptr(), M, K, T, variant, torch.cuda.current_stream().cuda_stream)
    return y


def _operands(M, K, T, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    Wq = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8, device="cuda")
    Xq = torch.randint(-127, 128, (T, K), generator=g, dtype=torch.int8, device="cuda")
    Wd = (torch.randn((M, K // 32), generator=g, device="cuda") * 0.02).half()
    Xd = (torch.rand((T, K // 32), generator=g, device="cuda") * 0.02).half()
    return Wq, Wd, Xq, Xd


# rows in shared memory: 16, 20, 24, 28 blocks; streamed: fewer than 16 lanes, one round, ragged last rounds, many rounds;
# rows and columns at the edges of tiles; several tiles per CTA, in the second case with a change of rows in between
SIZES = [(128, 512, 32), (127, 640, 31), (129, 768, 33), (1, 896, 1), (900, 896, 97), (19300, 896, 70), (128, 128, 9), (130, 256, 40),
         (1, 384, 3), (257, 1024, 32), (300, 1152, 33), (140, 2048, 129), (200, 4864, 65), (128, 14336, 32), (19300, 256, 70)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,T", SIZES)
def test_pair_gemm_bit_exact(oracle, M, K, T):
    Wq, Wd, x = synth.gemv_case(M, K, T=T, seed=M + T)
    dWq, dWd = torch.from_numpy(np.ascontiguousarray(Wq)).cuda(), torch.from_numpy(np.ascontiguousarray(Wd).view(np.int16)).cuda()
    dx = torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()
    xq, xd = torch.empty((T, K), dtype=torch.int8, device="cuda"), torch.empty((T, K // 32), dtype=torch.int16, device="cuda")
    _lib.call("lt_quant_q8", dx.data_ptr(), xq.data_ptr(), xd.data_ptr(), K, T, torch.cuda.current_stream().cuda_stream)
    want = oracle.q8_gemm(Wq, Wd, xq.cpu().numpy().reshape(-1), xd.cpu().numpy().view(np.uint16).reshape(-1), M, K, T).reshape(T, M)
    rng = np.random.default_rng(5)
    bias, R = rng.standard_normal(M).astype(np.float32), rng.standard_normal((T, M)).astype(np.float32)
    for resid, ld, w in ((None, 0, want), (bias, 0, want + bias), (R, M, want + R)):
        y = _gemm(dWq, dWd, xq, xd, M, K, T, 6, None if resid is None else torch.from_numpy(resid).cuda(), ld).cpu().numpy()
        assert np.array_equal(y.view(np.uint32), w.astype(np.float32).view(np.uint32))
    assert _lib.device_status() == set()


@pytest.mark.gpu
@pytest.mark.parametrize("K", [896, 1152])
def test_pair_gemm_unusual_scales(K):
    """Scales that are zero, subnormal, the largest, infinite or NaN, in weights and activations: the bits of the 16-column
    tiles, which multiply them one by one; so also with scales that start at an odd multiple of two bytes."""
    M, T = 300, 70
    Wq, Wd, Xq, Xd = _operands(M, K, T, 3)
    for t, rows in ((Wd, M), (Xd, T)):
        flat = t.view(-1)
        for i, v in enumerate((0.0, 6e-8, 6.1e-5, 65504.0, -65504.0)):
            flat[37 * i + 5::911] = v
    Wd[17, 3], Wd[130, 20], Wd[131, 0], Wd[299, 27], Xd[3, 11], Xd[40, 2] = float("inf"), float("nan"), float("-inf"), float("inf"), float("inf"), float("nan")
    Wq[17, 96:128] = 0                                         # infinity times an empty sum
    for shift in (0, 1):
        pad = [torch.zeros(t.numel() + 1, dtype=torch.float16, device="cuda") for t in (Wd, Xd)]
        for p, t in zip(pad, (Wd, Xd)):
            p[shift:shift + t.numel()] = t.reshape(-1)
        wd, xd = pad[0][shift:], pad[1][shift:]
        want, got = _gemm(Wq, Wd, Xq, Xd, M, K, T, 1), _gemm(Wq, wd, Xq, xd, M, K, T, 6)
        assert torch.equal(want.view(torch.int32), got.view(torch.int32)) and not torch.isfinite(want[0, 17])
    assert _lib.device_status() == set()


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,T", [(4096, 14336, 256), (1200, 896, 900)])
def test_pair_gemm_rows_with_an_infinite_scale(M, K, T):
    """A row in 128 with an infinite scale, one column with an infinite scale: the bits of the 16-column tiles, in at most five times the
    time (one thread per row and columns byte by byte took 67 times as long)."""
    Wq, Wd, Xq, Xd = _operands(M, K, T, 4)

    def us(variant):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(6)]
        for e in ev:
            y = _gemm(Wq, Wd, Xq, Xd, M, K, T, variant)
            e.record()
        torch.cuda.synchronize()
        return y, sorted(a.elapsed_time(b) for a, b in zip(ev, ev[1:]))[2]
    plain = us(6)[1]
    Wd[5::128, K // 64], Xd[T // 2, 1] = float("inf"), float("inf")
    got, odd = us(6)
    assert torch.equal(us(1)[0].view(torch.int32), got.view(torch.int32)) and not torch.isfinite(got[0, 5]) and torch.isfinite(got[0, 6])
    assert odd < 5 * plain + 0.05, (plain, odd)
    assert _lib.device_status() == set()
