"""The cross-entropy kernel waits with a limit: both callers hand it the device's status word to report to."""
import types

import torch

from ghost_flow_b200.ops import _lib, fused, raw


def _record(monkeypatch):
    calls, word = [], torch.zeros(8, dtype=torch.int32)
    monkeypatch.setattr(_lib, "cuda_lib", lambda: types.SimpleNamespace(gf_xent_fused=lambda *a: calls.append(a) or 0))
    monkeypatch.setattr(_lib, "status_word", lambda device=None: word)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: 77)
    return calls, word


def test_both_callers_pass_the_status_word(monkeypatch):
    calls, word = _record(monkeypatch)
    x, tg = torch.zeros(2, 64, dtype=torch.bfloat16), torch.tensor([1, 2])
    fused._XentFn.forward(types.SimpleNamespace(save_for_backward=lambda *a: None), x, tg, None, False)
    monkeypatch.setattr(raw, "_k", lambda t: True)
    raw.xent_fwd_bwd(x, tg)
    assert len(calls) == 2
    for a in calls:
        assert len(a) == len(_lib._SIGS["gf_xent_fused"]) and a[-2] == word.data_ptr() and a[-1] == 77
