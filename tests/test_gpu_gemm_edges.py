"""The slice-pair GEMM at the edges of its tiles, UMMA lists and conversions, held
bit for bit to the oracle: sizes one off the tile and the K step, schedules from two
slices up (a block with more bins than slices has no UMMA that spans it), results that
cancel to almost nothing, subnormal and overflowing results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ozlib, A, B, s, J, hint=None, bits=7):
    import torch
    dev = torch.device("cuda", 0)
    M, K = A.shape
    N = B.shape[1]
    dA, dB = torch.from_numpy(np.ascontiguousarray(A)).to(dev), torch.from_numpy(np.ascontiguousarray(B)).to(dev)
    dC = torch.full((M, N), float("nan"), dtype=torch.float64, device=dev)
    h = ozlib.Handle()
    h.set_bits(bits)
    h.set_slices(s)
    h.set_bins(J)
    if hint:
        h.set_plan_hint(**hint)
    for _ in range(2):  # the second call finds the first one's buffers
        rc = h.dgemm_device(M, N, K, dA.data_ptr(), K, dB.data_ptr(), N, dC.data_ptr(), N,
                            torch.cuda.current_stream().cuda_stream)
        assert rc == 0, h.last_error()
        assert h.sync() == 0, h.last_error()
    cfg = h.config()
    h.close()
    return dC.cpu().numpy(), cfg


def _same(got, ref, what):
    bad = np.argwhere(got.view(np.uint64) != ref.view(np.uint64))
    assert bad.size == 0, (what, bad[:4])


@pytest.mark.parametrize("s,J", [(2, 2), (2, 3), (3, 5), (4, 7), (5, 6), (8, 8), (8, 9), (8, 15), (10, 11), (12, 12),
                                 (16, 16)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 47, 15), (129, 49, 33), (130, 65, 161), (257, 97, 400)])
def test_edges_bit_exact(ozlib, oracle, s, J, M, N, K):
    A = oracle.gen_phi((M, K), 71, 1.0)
    B = oracle.gen_phi((K, N), 72, 1.0)
    got, cfg = _run(ozlib, A, B, s, J)
    _same(got, oracle.dgemm(A, B, 7, s, J, 0), cfg)


@pytest.mark.parametrize("s,J,blocks", [(2, 3, (3,)), (3, 5, (5,)), (3, 5, (4, 1))])
def test_block_with_more_bins_than_slices(ozlib, oracle, s, J, blocks):
    """No UMMA spans such a block: its accumulator is zeroed by the drain instead."""
    M, N, K = 150, 70, 1100
    A = oracle.gen_phi((M, K), 73, 1.0)
    B = oracle.gen_phi((K, N), 74, 1.0)
    got, cfg = _run(ozlib, A, B, s, J, dict(block_nb=blocks, tile_n=32))
    assert cfg["block_nb"][:cfg["blocks"]] == list(blocks)
    _same(got, oracle.dgemm(A, B, 7, s, J, 0), cfg)


@pytest.mark.parametrize("s,J", [(8, 8), (8, 15), (11, 12), (16, 16)])
@pytest.mark.parametrize("scale_a,scale_b", [(1.0, 1.0), (2.0 ** -540, 2.0 ** -530), (2.0 ** 520, 2.0 ** 505)])
def test_cancelling_and_out_of_range_results(ozlib, oracle, s, J, scale_a, scale_b):
    """A = [X, X], B = [Y; -Y + D]: most of the sum cancels, so the leading groups of
    the exact sum are zero or small; scaled results are subnormal or overflow."""
    M, N, K = 96, 64, 320
    X, Y = oracle.gen_phi((M, K), 75, 0.5), oracle.gen_phi((K, N), 76, 0.5)
    D = np.where(np.arange(N) % 3 == 0, 0.0, Y * 2.0 ** -(np.arange(N) % 52))
    A = np.concatenate([X, X], axis=1) * scale_a
    B = np.concatenate([Y, -(Y + D)], axis=0) * scale_b
    got, cfg = _run(ozlib, A, B, s, J)
    _same(got, oracle.dgemm(A, B, 7, s, J, 0), cfg)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("b,s,K", [(7, 8, 1000), (7, 8, 1100), (7, 12, 250), (7, 12, 300), (3, 18, 70), (3, 18, 301),
                                   (4, 9, 255)])
def test_one_launch_split_matches_two(ozlib, oracle, b, s, K, ta, tb):
    """Exponents and slices in one launch (short K) and in two: every operand order,
    padded odd leading dimensions, one and two windows, both carriers."""
    import torch
    M, N = 133, 49
    A, B = oracle.gen_phi((M, K), 77, 1.0), oracle.gen_phi((K, N), 78, 1.0)
    A[5] = 0.0
    B[:, 7] = 0.0
    dev = torch.device("cuda", 0)

    def stored(x, trans):
        x = np.ascontiguousarray(x.T if trans else x)
        buf = torch.full((x.shape[0], x.shape[1] + 3), float("nan"), dtype=torch.float64, device=dev)
        buf[:, :x.shape[1]] = torch.from_numpy(x)
        return buf

    dA, dB = stored(A, ta), stored(B, tb)
    dC = torch.full((M, N), float("nan"), dtype=torch.float64, device=dev)
    h = ozlib.Handle()
    h.set_bits(b)
    h.set_slices(s)
    h.set_bins(s)
    rc = h.dgemm_ex(ta, tb, M, N, K, 1.0, dA.data_ptr(), dA.shape[1], dB.data_ptr(), dB.shape[1], 0.0, dC.data_ptr(),
                    N, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, h.last_error()
    assert h.sync() == 0, h.last_error()
    h.close()
    _same(dC.cpu().numpy(), oracle.dgemm(A, B, b, s, s, 0), (b, s, K, ta, tb))


@pytest.mark.parametrize("s,J", [(8, 8), (8, 9), (8, 15), (11, 12)])
@pytest.mark.parametrize("M,N,K", [(140, 60, 1000), (130, 100, 3001)])
@pytest.mark.parametrize("kind", ["largest", "half", "one_row", "zero"])
def test_drains_that_follow_the_data(ozlib, oracle, s, J, M, N, K, kind):
    """Operands whose digits are all 2^7 - 1 and of one sign reach the fp32 bound that the
    drain periods are made for; operands that do so in some rows or columns of a tile
    only, or hold zeros, get longer periods elsewhere.  Bit-exact in every case, with one
    launch and with two for the stage kernels."""
    A, B = oracle.gen_phi((M, K), 81, 1.0), oracle.gen_phi((K, N), 82, 1.0)
    full = np.nextafter(1.0, 0.0)  # 53 ones: every digit 127
    if kind == "largest":
        A[:], B[:] = full, full
    elif kind == "half":
        A[: M // 2], B[:, ::2] = full, -full
    elif kind == "one_row":
        A[129, :], B[:, 17] = full, full
    else:
        A[:] = 0.0
        A[3, 5] = 1.5
    got, cfg = _run(ozlib, A, B, s, J)
    _same(got, oracle.dgemm(A, B, 7, s, J, 0), (cfg, kind))


@pytest.mark.parametrize("b,s,J", [(3, 25, 25), (3, 27, 27), (3, 29, 29), (2, 30, 30)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (129, 17, 33), (257, 33, 700), (300, 200, 1024)])
def test_slices_in_parts(ozlib, oracle, b, s, J, M, N, K):
    """Narrow slices whose stage fills shared memory come in parts of A's slices: K of
    one chunk and of many, tiles with one and with several units per SM."""
    A = oracle.gen_phi((M, K), 83, 1.0)
    B = oracle.gen_phi((K, N), 84, 1.0)
    got, cfg = _run(ozlib, A, B, s, J, bits=b)
    assert cfg["slice_format"] == 1
    _same(got, oracle.dgemm(A, B, b, s, J, 0), cfg)


@pytest.mark.parametrize("M,N,K,mode", [(96, 80, 200, 1), (256, 256, 2048, 1), (2304, 2000, 600, 0)])
def test_captured_call_replays(ozlib, M, N, K, mode):
    """A warmed-up call captured in a CUDA graph (one stage launch and two, with and
    without norms, the GEMM as a programmatic dependent) replays on new operands."""
    import torch
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(5)
    dA = torch.randn((M, K), dtype=torch.float64, device=dev, generator=gen)
    dB = torch.randn((K, N), dtype=torch.float64, device=dev, generator=gen)
    dC = torch.zeros((M, N), dtype=torch.float64, device=dev)
    h = ozlib.Handle()
    assert h.setup(M, N, K, mode) == 0, h.last_error()

    def call():
        rc = h.dgemm_device(M, N, K, dA.data_ptr(), K, dB.data_ptr(), N, dC.data_ptr(), N,
                            torch.cuda.current_stream().cuda_stream)
        assert rc == 0, h.last_error()

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call()
    for seed in (6, 7):
        gen.manual_seed(seed)
        dA.normal_(generator=gen)
        dB.normal_(generator=gen)
        dC.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        got = dC.clone()
        call()
        assert h.sync() == 0, h.last_error()
        assert torch.equal(got, dC)
    h.close()


@pytest.mark.parametrize("b,s,J,K", [(4, 18, 18, 9100), (4, 9, 9, 17000), (4, 13, 17, 9100), (4, 7, 7, 70), (2, 10, 11, 1500),
                                     (3, 18, 19, 1500)])
@pytest.mark.parametrize("kind", ["random", "largest"])
def test_two_blocks_dealt_to_three_issuers(ozlib, oracle, b, s, J, K, kind):
    """e4m3 plans of two bin blocks deal the UMMAs of both over the three issuing warps, all
    of them accumulating: several drains of each block in a tile, digits of 2^b - 1."""
    M, N = 133, 70
    A, B = oracle.gen_phi((M, K), 85, 1.0), oracle.gen_phi((K, N), 86, 1.0)
    if kind == "largest":
        A[:], B[:] = np.nextafter(1.0, 0.0), np.nextafter(1.0, 0.0)
    got, cfg = _run(ozlib, A, B, s, J, bits=b)
    assert (cfg["slice_format"], cfg["blocks"], cfg["issuers"]) == (1, 2, 3), cfg
    _same(got, oracle.dgemm(A, B, b, s, J, 0), cfg)
