"""Arguments that the few-row product and the one-call decoder layer refuse before they launch anything. The pointers are numbers
that nothing reads."""
import pytest
import torch

from ghost_flow_b200.ops import _lib, raw

BAD_ARG, P = -1, 1 << 20


def _rows(x=P, w=P, c=P, M=8, N=256, K=512, kind=1, norm=P, ldx=None):
    return _lib.cuda_lib().gf_gemm_rows(x, K if ldx is None else ldx, w, K, c, N, 0, M, N, K, kind, norm, 1e-6, None, None, 0, 1.0, 0, None, None)


@pytest.mark.parametrize("kw", [dict(norm=P + 2), dict(norm=P + 8), dict(norm=None), dict(x=P + 8), dict(w=P + 2), dict(kind=3),
                                dict(kind=-1), dict(M=17), dict(M=17, kind=2), dict(K=516), dict(ldx=516), dict(M=65, kind=0)])
def test_few_row_product(kw):
    assert _rows(**kw) == BAD_ARG


NAMES = "x attn_norm eps wqkv wo ffn_norm eps2 gate_up down cos sin kc vc s_max y ws B hidden inner Hq Hkv D inter pos splits".split()
VALUES = dict(dict.fromkeys(NAMES, P), eps=1e-6, eps2=1e-6, s_max=64, B=2, hidden=256, inner=512, Hq=4, Hkv=2, D=64, inter=0, pos=3,
              splits=1)


@pytest.mark.parametrize("kw", [
    *({n: P + 8} for n in "x attn_norm wqkv wo ffn_norm gate_up down kc vc y ws".split()), *({n: None} for n in ("kc", "cos", "ws")),
    dict(pos=64), dict(B=65), dict(B=0), dict(D=96), dict(hidden=260), dict(inner=516), dict(Hkv=3), dict(splits=0)])
def test_decoder_layer(kw):
    v = {**VALUES, **kw}
    assert _lib.cuda_lib().gf_llama_decode_layer(*(v[n] for n in NAMES), None, None) == BAD_ARG


@pytest.mark.parametrize("x,norm,w", [
    (torch.zeros(2, 64), torch.zeros(64), torch.zeros(8, 64)),                                    # fp32
    (*(torch.zeros(s, dtype=torch.bfloat16) for s in ((2, 64), (32,), (8, 64))),),
    (*(torch.zeros(s, dtype=torch.bfloat16) for s in ((2, 64), (64,), (8, 72))),),
    (torch.zeros(2, 128, dtype=torch.bfloat16)[:, ::2], *(torch.zeros(s, dtype=torch.bfloat16) for s in ((64,), (8, 64))))])
def test_norm_in_front_of_a_product(x, norm, w):
    with pytest.raises(ValueError, match="rmsnorm_gemm takes"):
        raw.rmsnorm_gemm(x, norm, 1e-6, w)
