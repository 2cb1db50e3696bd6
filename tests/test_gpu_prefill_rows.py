"""Rope, append and attention of the chunks of several sequences in one launch each: the bits of one sequence at a time."""
import ctypes

import pytest
import torch

from llamatov_b200 import _lib, dev_residency as dr, prefill, synth

pytestmark = pytest.mark.gpu


# short chunks (one at a time inside the call), score rows beside the tiles, blocks of 32 rows (also with one row over), as many
# sequences as a call takes; lengths before the chunk that differ, zero among them
@pytest.mark.parametrize("hd,nh,nkv,T,starts", [
    (64, 14, 2, 5, [0, 3]), (64, 14, 2, 33, [0, 40, 7]), (64, 14, 2, 333, [0, 0, 0]), (64, 14, 2, 353, [700, 0, 1]), (64, 4, 4, 64, [0, 1, 2, 3, 64, 65, 300, 9]),
    (128, 8, 2, 100, [0, 513]), (128, 32, 8, 225, [0, 100]), (64, 14, 2, 40, [12])])
def test_rows_of_sequences_bit_exact(hd, nh, nkv, T, starts):
    g = torch.Generator(device="cuda").manual_seed(T)
    st, f32, B, ld, width = torch.cuda.current_stream().cuda_stream, dict(device="cuda"), len(starts), (nh + 2 * nkv) * hd, nkv * hd
    X = torch.randn((B * T, ld), generator=g, **f32)
    caches = [[torch.randn((s + T + 5, width), generator=g, **f32) for _ in "kv"] for s in starts]
    scale, theta = hd ** -0.5, 1e6

    X1, want, kv1 = X.clone(), torch.empty((B * T, nh * hd), **f32), [[t.clone() for t in c] for c in caches]
    lens1 = torch.tensor(starts, dtype=torch.int32, device="cuda")
    for b, (k, v) in enumerate(kv1):
        rows, ln = X1[b * T:], lens1[b:].data_ptr()
        _lib.call("lt_rope_rows", rows.data_ptr(), ld, ln, T, nh + nkv, hd, theta, st)
        _lib.call("lt_append_kv_rows", k.data_ptr(), rows.data_ptr() + 4 * nh * hd, v.data_ptr(), rows.data_ptr() + 4 * (nh + nkv) * hd, ld, ln,
                  width, len(k), T, 1, st)
        _lib.call("lt_attn_prefill", rows.data_ptr(), ld, k.data_ptr(), v.data_ptr(), ln, want[b * T:].data_ptr(), nh * hd, hd, nh, nkv, scale, T,
                  starts[b] + T, st)

    got, lens = torch.full_like(want, float("nan")), torch.full_like(lens1, -1)
    seqs = _lib.RowSeqs()
    for b, (k, v) in enumerate(caches):
        seqs.k[b], seqs.v[b], seqs.len[b], seqs.start[b], seqs.max_seq[b] = k.data_ptr(), v.data_ptr(), lens[b:].data_ptr(), starts[b], len(k)
    _lib.call("lt_rope_append_rows", X.data_ptr(), ld, ctypes.byref(seqs), B, T, nh, nkv, hd, theta, st)
    _lib.call("lt_attn_prefill_rows", X.data_ptr(), ld, ctypes.byref(seqs), B, T, got.data_ptr(), nh * hd, hd, nh, nkv, scale, st)
    for a, b in [(X1, X), (want, got)] + [p for c in zip(kv1, caches) for p in zip(*c)]:
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert torch.equal(lens, lens1) and lens.tolist() == [s + T for s in starts]
    assert _lib.device_status() == set()


def test_rows_that_do_not_fit_are_refused():
    X = torch.zeros((4, 3 * 64), device="cuda")
    k, ln = torch.zeros((5, 64), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    seqs = _lib.RowSeqs()
    seqs.k[0], seqs.v[0], seqs.len[0], seqs.start[0], seqs.max_seq[0] = k.data_ptr(), k.data_ptr(), ln.data_ptr(), 2, 5
    for B in (1, 0, 9):
        with pytest.raises(RuntimeError):
            _lib.call("lt_rope_append_rows", X.data_ptr(), 192, ctypes.byref(seqs), B, 4, 1, 1, 64, 1e4, torch.cuda.current_stream().cuda_stream)


def test_one_cache_for_two_portions_of_a_batch():
    """The second portion continues the first one's context: the bits of one portion of both."""
    dr.reset_engine_state()
    dr.apply_production_profile()
    m = synth.make_model("tiny-qwen64", seed=3)
    w, cfg = synth.reference_weights(m)
    toks = torch.randint(0, m["cfg"]["vocab"], (2, 40), generator=torch.Generator().manual_seed(1))
    one, two = [None] * cfg["n_layers"], [None] * cfg["n_layers"]
    want = prefill.prefill_resident(w, cfg, toks.reshape(-1), one)
    got = prefill.prefill_resident(w, cfg, toks, [two, two])
    assert torch.equal(want.view(torch.int32), got.view(torch.int32))
    for a, b in zip(one, two):
        assert a.length == b.length == int(b._len.item()) == 80
        assert (a.k_slice_host() == b.k_slice_host()).all() and (a.v_slice_host() == b.v_slice_host()).all()
