"""Surrogate.forward on tensors that torch is still writing: the network reads
what the current stream's earlier work leaves, as any torch function does."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side_stream", [False, True])
def test_forward_waits_for_its_input(grrt, need_gpu, side_stream):
    import torch
    S = grrt.Surrogate(3)
    n = 5000
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(n, 4, device="cuda", generator=g)
    want = torch.empty(n, 16, device="cuda")
    torch.cuda.synchronize()
    S.forward(x, want, n)
    late = torch.full_like(x, 0.125)
    got = torch.empty(n, 16, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)  # about 10 ms before the input is there
        late.copy_(x)
        S.forward(late, got, n)
    torch.cuda.synchronize()
    assert torch.equal(got, want)


def test_forward_under_capture_runs_outside_the_graph(grrt, need_gpu):
    """As with pointers: the outputs are there when the call returns, and the
    capture of the program's other work goes on."""
    import torch
    S = grrt.Surrogate(3)
    n = 300
    x = torch.rand(n, 4, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    want, got, y = torch.empty(n, 16, device="cuda"), torch.zeros(n, 16, device="cuda"), torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    S.forward(x, want, n)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        y += 1
        S.forward(x, got, n)
        y += 1
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((y == 2).all())
