"""The library's count of its launches against the kernels that a captured call consists of."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernels(graph):
    from cuda.bindings import runtime as rt

    h = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    _, _, n = rt.cudaGraphGetNodes(h, 0)
    _, nodes, n = rt.cudaGraphGetNodes(h, n)
    return sum(rt.cudaGraphNodeGetType(v)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for v in nodes[:n])


def _randn(*s):
    return torch.randn(*s, device="cuda").bfloat16()


def _gpt(train):
    from ghost_flow_b200.models.configs import GPTConfig
    from ghost_flow_b200.models.gpt import GPTBlock

    m = GPTBlock(GPTConfig(n_embd=256, n_head=4, n_inner=512, dropout=0.0)).to(device="cuda", dtype=torch.bfloat16)
    x, dy = _randn(2, 128, 256).requires_grad_(train), _randn(2, 128, 256)
    return lambda: torch.autograd.grad(m(x), [x, *m.parameters()], dy) if train else m(x)


def _layer(B):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.models import LLaMAConfig
    from ghost_flow_b200.models.llama import LLaMADecoderLayer

    cfg = LLaMAConfig(vocab_size=64, hidden_size=256, intermediate_size=512, num_hidden_layers=1, num_attention_heads=4,
                      num_key_value_heads=2, max_position_embeddings=512)
    m = LLaMADecoderLayer(cfg, device="cuda", dtype=torch.bfloat16)
    cos, sin = ops.rope_tables(512, 64, 10000.0, "cuda")
    x, c = _randn(B, 1, 256), (_randn(B, 400, 2, 64), _randn(B, 400, 2, 64))
    return lambda: m(x, cos, sin, cache=c, start_pos=333)


def _product(M, N, K):
    from ghost_flow_b200 import ops

    a, b = _randn(M, K), _randn(N, K)
    return lambda: ops.matmul_nt(a, b)


def _norm():
    from ghost_flow_b200 import ops

    x, w = _randn(256, 1024).requires_grad_(), _randn(1024).requires_grad_()
    return lambda: torch.autograd.grad(ops.rms_norm(x, w), [x, w], x.detach())


def _attention():
    from ghost_flow_b200 import ops

    q, k, v = (_randn(2, 256, 4, 64).requires_grad_() for _ in range(3))
    return lambda: torch.autograd.grad(ops.flash_attention(q, k, v), [q, k, v], q.detach())


@pytest.mark.parametrize("make", [
    lambda: _gpt(False), lambda: _gpt(True), lambda: _layer(2), lambda: _layer(40), _norm, _attention,
    # few rows on either kernel, whole tiles of a CTA and of a pair, sums of parts of K in both forms
    lambda: _product(4, 512, 512), lambda: _product(16, 4096, 4096), lambda: _product(256, 256, 256), lambda: _product(4096, 4096, 512),
    lambda: _product(768, 768, 8192), lambda: _product(3072, 768, 8192)],
    ids="gpt gpt-train layer-2 layer-40 norm attention skinny rows tile pair sums slices".split())
def test_count_is_the_kernels_of_a_call(make, kernel_status):
    from ghost_flow_b200.ops import _lib

    f, graph = make(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.set_grad_enabled("grad" in f.__code__.co_names):
        f()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            n = _lib.launch_count()
            f()
            n = _lib.launch_count() - n
    assert n == _kernels(graph)
