"""Loading weights into a network that has captured graphs: its bf16 copies
stay where the graphs read and write them, and hold the loaded weights."""
import pytest
import torch

from pca_gb300.valuenet import LAYERS, ValueNet


def host_net(seed):
    """The parameters of a network, on the host (no kernels)."""
    net = object.__new__(ValueNet)
    g = torch.Generator().manual_seed(seed)
    net.dev = torch.device("cpu")
    net.W = {n: torch.rand(o, i, generator=g) - 0.5 for n, o, i in LAYERS}
    net.b = {n: torch.rand(o, generator=g) - 0.5 for n, o, i in LAYERS}
    net.Wb, net.Wt = {}, {}
    net._refresh_bf16()
    return net


def test_loaded_weights_keep_their_place():
    net, other = host_net(1), host_net(2)
    tensors = [d[n] for d in (net.W, net.b, net.Wb, net.Wt) for n, _, _ in LAYERS]
    places = [t.data_ptr() for t in tensors]
    net.load_state_dict(other.state_dict())
    assert [d[n].data_ptr() for d in (net.W, net.b, net.Wb, net.Wt)
            for n, _, _ in LAYERS] == places
    for n, out, inp in LAYERS:
        assert torch.equal(net.W[n], other.W[n]) and torch.equal(net.b[n], other.b[n])
        assert torch.equal(net.Wb[n], other.W[n].to(torch.bfloat16))
        assert torch.equal(net.Wt[n], other.W[n].t().to(torch.bfloat16))
        assert net.Wb[n].is_contiguous() and net.Wt[n].is_contiguous()
        assert net.Wt[n].shape == (inp, out)


def batch(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ri = lambda lo, hi, shape: torch.randint(lo, hi, shape, generator=g, device="cuda",  # noqa: E731
                                             dtype=torch.int32)
    regs = ri(0, 1 << 16, (n, 8, 32))
    regs[:, 0] = 0
    return dict(regs=regs.to(torch.int16), flags=ri(0, 16, (n, 32)).to(torch.uint8),
                live=ri(0, 256, (n,)).to(torch.uint8), task=ri(0, 3, (n,)).to(torch.int16),
                task_io=ri(0, 1 << 16, (3, 3, 32)).to(torch.int16), task_T=ri(16, 33, (3,)),
                depth=ri(1, 5, (n,)).to(torch.uint8), label=(ri(0, 2, (n,)) > 0).float(),
                remaining=ri(1, 4, (n,)), TP=32)


@pytest.mark.gpu
def test_a_graph_captured_before_the_load_trains_the_loaded_weights():
    data, weights = [batch(256, s) for s in range(4)], ValueNet(seed=9).state_dict()
    plain, graph = ValueNet(seed=1), ValueNet(seed=1)
    for b in data[:2]:   # the second call replays the captured step
        plain.train_step(b)
        graph.train_step_graph(b)
    for net in (plain, graph):
        net.load_state_dict(weights)
    for b in data[2:]:
        assert torch.equal(plain.train_step(b), graph.train_step_graph(b))
    for d, e in ((plain.W, graph.W), (plain.b, graph.b), (plain.Wb, graph.Wb),
                 (plain.Wt, graph.Wt), (plain.mW, graph.mW)):
        for n, _, _ in LAYERS:
            assert torch.equal(d[n], e[n])
    b = data[3]
    states = (b["regs"], b["flags"], b["live"], b["task"], b["depth"], 32, b["task_io"],
              b["task_T"])
    assert torch.equal(plain.forward_fused(*states), graph.forward_fused(*states))
    plain.check_status()
    graph.check_status()
