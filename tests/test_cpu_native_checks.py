"""What the wrappers of the native kernels look at before they pass an address on: an operand on another device, or one
that the kernel's wide loads could not read, never reaches a launch.  The native library is replaced by a recorder."""
import os
import re

import pytest
import torch

import genesis_b200  # noqa: F401
from genesis_b200.ops import dispatch as K
from genesis_b200.ops import native as N


class _Elsewhere(torch.Tensor):
    """A tensor of another device, as far as the wrappers look."""
    def get_device(self):
        return 5


def _elsewhere(t):
    return t.as_subclass(_Elsewhere)


class _Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 0
        return call


@pytest.fixture
def native(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(N, "lib", lambda: rec)
    monkeypatch.setattr(N, "_st", lambda: 0)
    monkeypatch.setattr(N, "status_tensor", lambda dev: torch.zeros(8, dtype=torch.int32))
    return rec


def test_stacked_conversion_takes_one_device_and_whole_rows(native):
    a, b = torch.randn(4, 8), torch.randn(2, 8)
    out = torch.empty(6, 8, dtype=torch.bfloat16)
    assert N.cast_stack([a, b], out) is out and native.calls == ["gb_cast_stack"]
    native.calls.clear()
    for ts in ([a, _elsewhere(b)], [_elsewhere(a), b], [a, torch.randn(4, 4)], [a, torch.randn(16)], [a, torch.randn(1, 8)]):
        assert N.cast_stack(ts, out) is NotImplemented
    assert native.calls == []
    # rows that do not match are refused by the copies, as a concatenation would
    with pytest.raises(RuntimeError):
        K.cat_cast([a, torch.randn(4, 4)], torch.bfloat16)


@pytest.mark.parametrize("away", ["cos", "sin", "positions"])
def test_rotation_tables_of_another_device(native, away):
    B, S, Hq, Hkv, D = 2, 5, 2, 1, 8
    t = {"cos": torch.randn(16, D), "sin": torch.randn(16, D), "positions": torch.arange(S)}
    y, q, kv = torch.randn(B, S, (Hq + 2 * Hkv) * D), torch.randn(B, S, Hq, D), torch.randn(B, S, Hkv, D)

    def launches():
        native.calls.clear()
        r = (N.rope(q, t["cos"], t["sin"], t["positions"], False),
             N.qkv_rope(y, None, None, None, t["cos"], t["sin"], t["positions"], Hq, Hkv, D, False),
             N.qkv_rope(None, q, kv, kv, t["cos"], t["sin"], t["positions"], Hq, Hkv, D, True))
        return [x is NotImplemented for x in r], len(native.calls)

    assert launches() == ([False] * 3, 3)
    t[away] = _elsewhere(t[away])
    assert launches() == ([True] * 3, 0)


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
def test_norm_weights_that_the_kernels_cannot_read(native, monkeypatch, wdt):
    monkeypatch.setattr(N, "_colsum", lambda *a: None)
    rows, cols = 3, 16
    x, rstd = torch.randn(rows, cols).bfloat16(), torch.ones(rows)
    monkeypatch.setattr(_Recorder, "gb_rmsnorm_bwd_ctas", lambda *a: 1, raising=False)
    monkeypatch.setattr(_Recorder, "gb_norm_bwd_ctas", lambda *a: 1, raising=False)

    def refused(w):
        native.calls.clear()
        r = (N.rmsnorm_fwd(x, w, 1e-6), N.add_rmsnorm_fwd(x, x, w, 1e-6), N.rmsnorm_bwd(x, x, w, rstd),
             N.add_rmsnorm_bwd(x, x, x, w, rstd), N.layernorm_fwd(x, w, None, 1e-6), N.layernorm_fwd(x, None, w, 1e-6),
             N.layernorm_bwd(x, x, w, rstd, rstd))
        return {y is NotImplemented for y in r}, len(native.calls)

    base = torch.ones(2 * cols + 8, dtype=wdt)
    assert base.data_ptr() % 16 == 0
    assert refused(base[:cols]) == ({False}, 7)
    for w in (base[1:cols + 1], base[:2 * cols:2], _elsewhere(base[:cols]), base[:cols - 1], base[:1]):
        assert refused(w) == ({True}, 0)


def _kernels():
    """(file, head, body) of every kernel in the sources."""
    d = os.path.join(os.path.dirname(genesis_b200.__file__), "csrc")
    for f in sorted(os.listdir(d)):
        if f.endswith((".cu", ".cuh")):
            src = open(os.path.join(d, f)).read()
            for part in src.split("__global__ ")[1:]:
                body = part[:part.index("\n}")]
                yield f, " ".join(body[:120].split()), body


def test_kernels_that_give_up_wait_for_their_copies():
    """A kernel whose copies complete on barriers (its waits are bounded) lets the copies in flight land before it leaves.
    The path cannot be provoked by a sound kernel, so this looks at the sources."""
    seen = 0
    for f, name, body in _kernels():
        if "mbar_expect_tx(" in body or "ring.issue(" in body:
            seen += 1
            assert "drain_copies(" in body or "ring.drain(" in body, (f, name)
        # a barrier is always past one of its two parities, so a wait for either of them ends at once
        assert not re.search(r"!mbar_try_wait\(&?([^,]+), 0\) && !mbar_try_wait\(&?\1, 1\)", body), (f, name)
    assert seen >= 9


def test_stream_handle_without_torchs_private_names(monkeypatch):
    class Stream:
        cuda_stream = 7
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: Stream)
    raw, device = (lambda d: 100 + d), (lambda: 3)
    assert N._stream_handle(raw, device)() == 103
    assert N._stream_handle(None, device)() == 7 and N._stream_handle(raw, None)() == 7
