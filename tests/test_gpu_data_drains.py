"""Products whose drains follow the data (the split takes the slices' norms): their
buffers."""
import pytest

pytestmark = pytest.mark.gpu


def test_first_call_after_setup_can_be_captured(ozlib):
    """ozgb_setup reserves every buffer that a call of its shape fills, the slices' norms
    among them: the handle's first call allocates nothing and can be captured."""
    import torch
    dev = torch.device("cuda", 0)
    M, N, K = 2304, 2000, 2048
    gen = torch.Generator(device=dev).manual_seed(9)
    dA = torch.randn((M, K), dtype=torch.float64, device=dev, generator=gen)
    dB = torch.randn((K, N), dtype=torch.float64, device=dev, generator=gen)
    dC = torch.zeros((M, N), dtype=torch.float64, device=dev)

    def call(h):
        rc = h.dgemm_device(M, N, K, dA.data_ptr(), K, dB.data_ptr(), N, dC.data_ptr(), N,
                            torch.cuda.current_stream().cuda_stream)
        assert rc == 0, h.last_error()

    h = ozlib.Handle()  # loads the kernels
    call(h)
    assert h.sync() == 0, h.last_error()
    h.close()
    ref = dC.clone()
    h = ozlib.Handle()
    assert h.setup(M, N, K, 1) == 0, h.last_error()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call(h)
    dC.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(dC, ref)
    h.close()
