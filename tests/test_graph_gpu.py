"""A whole forward + backward of the Metis layer captured into a CUDA graph (fp4_post_b200.graphs):
the replay must compute what the eager step computes, follow the static inputs, and draw fresh
stochastic-rounding bits on every replay (the Philox offset lives on the device)."""
import pytest
import torch

import fp4_post_b200
from fp4_post_b200 import ops
from fp4_post_b200.graphs import GraphedStep

fp4_post_b200.install_reference_aliases()

from Metis.Metis.bitlinear import BitLinear, LinearLowbitFunction  # noqa: E402
from Metis.Metis.quant import Cast2NVFp4e2m1Block  # noqa: E402
from grpo.grpo import MetisArgs  # noqa: E402
from gpu_helpers import rel_l2  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module", autouse=True)
def _lib(built_library):
    return built_library


def make_layer(cache):
    torch.manual_seed(7)
    args = MetisArgs(forward_svd_rank=64, activation_lowrank_svd=64, backward_lowrank_svd=64, cache_quantized_weight=cache)
    args.device = DEV
    layer = BitLinear(512, 384, args=args, bias=True, dtype=torch.bfloat16, compute_dtype=torch.bfloat16)
    layer.layer_name = "graphed"
    layer.split()
    return layer.to(DEV)


def test_replay_matches_eager_follows_the_inputs_and_redraws_the_rounding_bits():
    layer = make_layer(cache=False)          # weight quantization inside the graph: safe when weights change
    assert LinearLowbitFunction.q_backward_outputgrad is Cast2NVFp4e2m1Block      # stochastic backward (GRPO default)
    params = list(layer.parameters())
    x = torch.randn(2, 256, 512, device=DEV, dtype=torch.bfloat16).requires_grad_(True)
    g = torch.randn(2, 256, 384, device=DEV, dtype=torch.bfloat16)

    def step():
        for p in params:
            p.grad = None
        x.grad = None
        y = layer(x)
        y.backward(g)
        return y, x.grad, layer.warmup_linear.weight.grad

    graphed = GraphedStep(step)
    y1, gx1, gw1 = (t.clone() for t in graphed())
    y2, gx2, gw2 = (t.clone() for t in graphed())
    y_e, gx_e, gw_e = (t.clone() for t in step())
    # forward: round to nearest everywhere, so eager and both replays agree bit for bit
    assert torch.equal(y1, y2) and torch.equal(y1, y_e)
    # backward: stochastic rounding with a fresh Philox offset per call, in replays too
    assert not torch.equal(gx1, gx2) and not torch.equal(gw1, gw2)
    for a in (gx1, gx2):
        assert rel_l2(a.float().cpu().numpy(), gx_e.float().cpu().numpy()) <= 0.2
    for a in (gw1, gw2):
        assert rel_l2(a.float().cpu().numpy(), gw_e.float().cpu().numpy()) <= 0.2

    # new contents of the static input tensors, same graph
    with torch.no_grad():
        x.copy_(torch.randn_like(x))
        g.copy_(torch.randn_like(g))
    y3 = graphed()[0].clone()
    assert not torch.equal(y3, y1)
    assert torch.equal(y3, step()[0])

    # the weights changed: with the cache off the replay re-quantizes them
    with torch.no_grad():
        layer.warmup_linear.weight.mul_(1.5)
    y4 = graphed()[0].clone()
    assert torch.equal(y4, step()[0]) and not torch.equal(y4, y3)


def test_stochastic_quantizer_counter_advances_once_per_call():
    ctr = torch.full((1,), 5, dtype=torch.int64, device=DEV)
    x = torch.randn(64, 256, device=DEV, dtype=torch.bfloat16)
    a = ops.nvfp4_quantize(x, stochastic=True, seed=1, offset_counter=ctr)
    b = ops.nvfp4_quantize(x, stochastic=True, seed=1, offset_counter=ctr)
    torch.cuda.synchronize()
    assert ctr.item() == 7
    assert not torch.equal(a.codes, b.codes)
    # the same bits as the host-side offset of the same value
    c = ops.nvfp4_quantize(x, stochastic=True, seed=1, offset=5)
    assert torch.equal(a.codes, c.codes) and torch.equal(a.scales, c.scales)
    with pytest.raises(ValueError):
        ops.nvfp4_quantize(x, stochastic=True, offset_counter=torch.zeros(1, dtype=torch.int32, device=DEV))


def test_light_stream_helpers_agree_with_torch():
    from fp4_post_b200 import ops
    dev = torch.device("cuda", torch.cuda.current_device())
    st, before = torch.cuda.Stream(device=dev), torch.cuda.current_stream(dev)
    assert ops.current_stream(dev) == before
    with pytest.raises(KeyError):
        with ops.on_stream(st):
            assert torch.cuda.current_stream(dev) == st == ops.current_stream(dev)
            with ops.on_stream(before):
                assert ops.current_stream(dev) == before
            assert ops.current_stream(dev) == st
            raise KeyError
    assert torch.cuda.current_stream(dev) == before


def _kernel_nodes(fn):
    """Kernel nodes of a captured call of fn."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        keep = fn()                                                    # noqa: F841
    handle = runtime.cudaGraph_t(graph.raw_cuda_graph())
    err, _, count = runtime.cudaGraphGetNodes(handle)
    assert int(err) == 0
    err, nodes, _ = runtime.cudaGraphGetNodes(handle, count)
    assert int(err) == 0
    kinds = [runtime.cudaGraphNodeGetType(n)[1] for n in nodes[:count]]
    graph.reset()
    return sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.parametrize("M,N,r", [(1120, 4096, 128), (19000, 512, 64), (64, 1024, 32)])       # several splits, one, several
def test_the_launch_counter_counts_the_kernels_of_the_low_rank_backward(M, N, r):
    g, u = torch.randn(M, N, device=DEV).to(torch.bfloat16), torch.randn(N, r, device=DEV).to(torch.bfloat16)
    yv, s = torch.randn(M, r, device=DEV).to(torch.bfloat16), torch.ones(r, device=DEV)
    for fn in (lambda: ops.lowrank_dts(g, u, yv, s), lambda: ops.lowrank_dts(g, u, yv, s, want_mean=True), lambda: ops.lowrank_du(g, yv)):
        before = ops.launch_count()
        nodes = _kernel_nodes(fn)
        assert ops.launch_count() - before == 2 * nodes                # an eager call and the captured one


@pytest.mark.parametrize("M,N,K", [(16, 128, 4096), (16, 4096, 14336), (5, 256, 256), (300, 128, 512)])        # split twice, not split twice
def test_the_launch_counter_counts_the_kernels_of_a_product(M, N, K):
    a, b = ops.nvfp4_quantize(torch.randn(M, K, device=DEV)), ops.nvfp4_quantize(torch.randn(N, K, device=DEV))
    s, one = torch.ones(N, device=DEV), torch.ones(1, device=DEV)
    for fn in (lambda: ops.nvfp4_gemm(a, b), lambda: ops.nvfp4_gemm(a, b, scaled=(s, one, one))):
        before = ops.launch_count()
        nodes = _kernel_nodes(fn)
        assert ops.launch_count() - before == 2 * nodes
