"""Host side of a prompt portion of the Q8_0 block, the library replaced by a recorder: which rows go to which cache in which launch,
and what the caches' lengths are afterwards."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from llamatov_b200 import _lib, archs, dev_residency as dr

T, HD, E, F, MAX_SEQ = 5, 64, 128, 256, 40
CFG = dict(n_embd=E, n_head=2, n_head_kv=1, norm_eps=1e-5, rope_theta=1e4)
W = {"blk.0.attn_norm.weight": 0, "blk.0.ffn_norm.weight": 0, "blk.0.attn_output.weight": (E, E), "blk.0.ffn_down.weight": (E, F)}


class Cache:
    def __init__(self, n, length):
        self.k_ptr, self.v_ptr, self.len_ptr, self.width, self.max_seq, self.length = 1000 * n, 1000 * n + 1, 1000 * n + 2, HD, MAX_SEQ, length

    def _ensure_len_ptr(self, seed=True):
        return self.len_ptr


@pytest.fixture
def run(monkeypatch):
    """run(caches, refuse): a layer over them; the launches over rows as (name, [(k, start)], first row)."""
    monkeypatch.setattr(dr, "_weights", lambda w: (0, 0, *w))
    monkeypatch.setattr(dr, "_fused_qkv_weight", lambda w, p: ((2 * E, E), None, None))
    monkeypatch.setattr(dr, "_fused_gateup_weight", lambda w, p: ((2 * F, E), None, (F, F)))
    for name, f in (("_np", lambda x: x), ("_dev_const", lambda x: 0), ("_vp", lambda x: x), ("_stream", lambda: 0), ("_capturing", lambda: False)):
        monkeypatch.setattr(dr, name, f)

    def layer(caches, refuse=None):
        B = len(caches)
        st = SimpleNamespace(w=W, cfg=CFG, B=B, T=T, R=B * T, F=F, **{n: torch.zeros(B * T, 2 * F) for n in ("x", "x1", "h", "qkv", "att", "gu", "xq", "xd")})
        seen = []

        def call(name, *a):
            if name == refuse:
                raise RuntimeError(name)
            if name in ("lt_rope_append_rows", "lt_attn_prefill_rows"):
                s = a[2]._obj
                base, width = (st.qkv.data_ptr(), 2 * E)
                seen.append((name[3:7], [(s.k[i], s.start[i]) for i in range(a[3])], (a[0] - base) // (4 * width)))
        monkeypatch.setattr(_lib, "call", call)
        archs.of(CFG).layer_rows(st, SimpleNamespace(layer=0, slot=0), caches)
        return seen
    return layer


def test_lengths_stay_where_the_append_is_refused(run):
    caches = [Cache(i + 1, i) for i in range(3)]
    with pytest.raises(RuntimeError, match="lt_rope_append_rows"):
        run(caches, refuse="lt_rope_append_rows")
    assert [c.length for c in caches] == [0, 1, 2]
    with pytest.raises(RuntimeError, match="lt_attn_prefill_rows"):      # the rows are in the caches
        run(caches, refuse="lt_attn_prefill_rows")
    assert [c.length for c in caches] == [T, T + 1, T + 2]


def test_ten_sequences_take_two_launches(run):
    caches = [Cache(i + 1, i) for i in range(10)]
    seen = run(caches)
    a, b = [(1000 * (i + 1), i) for i in range(8)], [(9000, 8), (10000, 9)]
    assert seen == [("rope", a, 0), ("attn", a, 0), ("rope", b, 8 * T), ("attn", b, 8 * T)]
    assert [c.length for c in caches] == [i + T for i in range(10)]


def test_a_cache_that_comes_again_goes_on_behind_its_rows(run):
    a, b = Cache(1, 3), Cache(2, 0)
    seen = run([a, b, a, a])
    assert [s for s in seen if s[0] == "rope"] == [("rope", [(1000, 3), (2000, 0)], 0), ("rope", [(1000, 3 + T)], 2 * T), ("rope", [(1000, 3 + 2 * T)], 3 * T)]
    assert [n for n, *_ in seen] == ["rope", "attn"] * 3 and (a.length, b.length) == (3 + 3 * T, T)


def test_the_library_refuses_one_length_for_two_sequences():
    s = _lib.RowSeqs()
    for i in range(2):
        s.k[i] = s.v[i] = s.len[i] = 4096 * (i + 1)
        s.max_seq[i] = MAX_SEQ
    s.len[1] = s.len[0]
    with pytest.raises(RuntimeError, match="one length"):
        _lib.call("lt_rope_append_rows", 4096, 192, ctypes.byref(s), 2, T, 1, 1, 64, 1e4, None)
