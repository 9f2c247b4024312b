"""Products whose drains follow the data (the split takes the slices' norms), held bit
for bit to the oracle on operands that reach the fp32 bound; the norms themselves; their
buffers, and what the autotuner times of them.  They have more than 304 tiles (smaller
products, test_gpu_gemm_edges.py's among them, drain by the worst case): the shapes here
have them in one direction, or in both.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FULL = float(np.nextafter(1.0, 0.0))  # 53 ones: every digit of the first 7 slices is 127


def _shapes(s, J, bn):
    """(M, N, K, stage launches before the GEMM): one launch for exponents and slices, or
    one for the exponents and one for each operand's slices."""
    side = 18 if bn >= 48 else 17
    n = (305 // side + 1) * bn - 7
    # past the one-launch limit: K > 2048, or for two windows 4 per block of the launch
    # (2284 x 809: 1356, 2156 x 569: 1232)
    both = [(2100, 3)] if s * 7 <= 63 else [(1300, 1 if bn >= 48 else 3), (1500, 3)]
    return [(100, 309 * bn + 5, 420, 1), (128 * 309 + 9, bn - 3, 420, 1)] + [(side * 128 - 20, n, k, x) for k, x in both]


def _plant(A, B, kind):
    """Operands as op(A), op(B) on the device: tiles whose digits are all 127 (of one sign),
    some rows and columns of a tile, one row and one column of all tiles, zeros."""
    if kind == "largest":
        A.fill_(FULL)
        B.fill_(FULL)
    elif kind == "half":
        A[: A.shape[0] // 2] = FULL
        B[:, ::2] = -FULL
    elif kind == "one_row":
        A[A.shape[0] // 2] = FULL
        B[:, B.shape[1] // 2] = FULL
    else:
        A.zero_()
        A[A.shape[0] // 3, 5] = 1.5
        B[:, : B.shape[1] // 2] = 0.0


def _samples(n, tile):
    """Both sides of the tiles' edges, the planted units and their neighbours."""
    at = [0, 1, n // 3, n // 2 - 1, n // 2, n // 2 + 1, n - 2, n - 1]
    at += [t * tile + d for t in (1, 2, n // tile // 2, n // tile) for d in (-1, 0)]
    return sorted({i for i in at if 0 <= i < n})


@pytest.mark.parametrize("kind", ["largest", "half", "one_row", "zero"])
@pytest.mark.parametrize("s,J", [(5, 5), (8, 8), (8, 9), (8, 15), (9, 9), (10, 10), (11, 12), (12, 12), (16, 16)])
def test_data_drains_bit_exact(ozlib, oracle, s, J, kind):
    """One and two windows, 32- and 16-deep chunks, BN = 64, 48 and 32, one stage launch and
    three, every operand order.  Digits of 127 and one sign make every bound tight: a
    period that is one chunk too long loses bits of odd sums past 2^24."""
    import torch
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(100 * s + J)
    bn = ozlib.plan_query(4096, 4096, 4096, 7, s, J)["tile_n"]
    for M, N, K, stages in _shapes(s, J, bn):
        assert ozlib.plan_data_drains(M, N, K, 7, s, J), (M, N, K)
        A = torch.randn((M, K), dtype=torch.float64, device=dev, generator=gen).exp_()
        B = torch.randn((K, N), dtype=torch.float64, device=dev, generator=gen).exp_()
        A *= torch.rand(A.shape, dtype=torch.float64, device=dev, generator=gen) - 0.5
        B *= torch.rand(B.shape, dtype=torch.float64, device=dev, generator=gen) - 0.5
        _plant(A, B, kind)
        rows, cols = _samples(M, 128), _samples(N, bn)
        ref = oracle.dgemm(np.ascontiguousarray(A[rows].cpu().numpy()),
                           np.ascontiguousarray(B[:, cols].cpu().numpy()), 7, s, J, 0)
        dC = torch.empty((M, N), dtype=torch.float64, device=dev)
        for ta in (0, 1):
            for tb in (0, 1):
                dA, dB = (A.T.contiguous() if ta else A), (B.T.contiguous() if tb else B)
                dC.fill_(float("nan"))
                h = ozlib.Handle()
                h.set_slices(s)
                h.set_bins(J)
                rc = h.dgemm_ex(ta, tb, M, N, K, 1.0, dA.data_ptr(), dA.shape[1], dB.data_ptr(), dB.shape[1], 0.0,
                                dC.data_ptr(), N, torch.cuda.current_stream().cuda_stream)
                assert rc == 0, h.last_error()
                assert h.sync() == 0, h.last_error()
                assert h.launch_count() == stages + 1
                h.close()
                got = dC[rows][:, cols].cpu().numpy()
                bad = np.argwhere(got.view(np.uint64) != ref.view(np.uint64))
                assert bad.size == 0, (M, N, K, ta, tb, bad[:4])


def _digits(torch, x, s):
    """Squares of the 7-bit digits of x (units along dimension 0), s x units x K, from the
    values: x / 2^(E - 1022) has the digits after the point, E a unit's largest exponent."""
    e = torch.frexp(x.abs().amax(dim=1, keepdim=True))[1]
    r = torch.ldexp(x.abs(), -e)
    out = []
    for _ in range(s):
        r = r * 128.0
        d = torch.floor(r)
        r = r - d
        out.append((d * d).float())
    return out


@pytest.mark.parametrize("kind", ["random", "largest"])
@pytest.mark.parametrize("s,J", [(5, 5), (7, 7), (8, 9), (9, 9), (8, 15), (10, 10), (12, 12), (16, 16)])
def test_norms_are_the_digits_own(ozlib, s, J, kind):
    """The norms that the drains are planned from, of every tile and slice, against the
    digits of the operands: equal, or up to twice where a kernel bounds a chunk by its
    larger half.  One that is too small would let fp32 sums
    pass 2^24."""
    import torch
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(7 * s + J)
    c = ozlib.plan_query(4096, 4096, 4096, 7, s, J)
    bn, kc = c["tile_n"], c["k_chunk"]
    for M, N, K, stages in _shapes(s, J, bn):
        A = torch.rand((M, K), dtype=torch.float64, device=dev, generator=gen) + 2.0 ** -20
        B = torch.rand((K, N), dtype=torch.float64, device=dev, generator=gen) + 2.0 ** -20
        if kind == "largest":
            A.fill_(FULL)
            B.fill_(FULL)
        want = []
        for x, tile in ((A, 128), (B.T, bn)):
            units, pad = x.shape[0], -x.shape[0] % tile
            per = []
            for d in _digits(torch, x, s):
                d = torch.nn.functional.pad(d, (0, -K % kc)).reshape(units, -1, kc).sum(dim=2).amax(dim=1)
                per.append(torch.nn.functional.pad(d, (0, pad)).reshape(-1, tile).amax(dim=1))
            want.append(torch.stack(per, dim=1))
        dC = torch.empty((M, N), dtype=torch.float64, device=dev)
        for ta in (0, 1):
            for tb in (0, 1):
                dA, dB = (A.T.contiguous() if ta else A), (B.T.contiguous() if tb else B)
                h = ozlib.Handle()
                h.set_slices(s)
                h.set_bins(J)
                for _ in range(2):
                    rc = h.dgemm_ex(ta, tb, M, N, K, 1.0, dA.data_ptr(), dA.shape[1], dB.data_ptr(), dB.shape[1], 0.0,
                                    dC.data_ptr(), N, torch.cuda.current_stream().cuda_stream)
                    assert rc == 0, h.last_error()
                    assert h.sync() == 0, h.last_error()
                tiles = [w.shape[0] for w in want]
                got = torch.from_numpy(h.last_norms(s * sum(tiles))).to(dev)
                h.close()
                parts = [got[: s * tiles[0]].reshape(-1, s), got[s * tiles[0]:].reshape(-1, s)]
                for side, (g, w) in enumerate(zip(parts, want)):
                    assert bool((g >= w).all()), (M, N, K, ta, tb, side, (g < w).sum(dim=0).tolist())
                    top = 2 * w if stages == 1 else w
                    assert bool((g <= top).all()), (M, N, K, ta, tb, side, (g > top).sum(dim=0).tolist())


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


def test_autotune_times_the_drains_that_calls_run(ozlib):
    """The autotuner takes the norms where a call of its plan does, so that the handle holds
    every buffer of such a call afterwards: it can be captured, with nothing allocated."""
    import torch

    from ozaie_gb300 import api
    dev = torch.device("cuda", 0)
    M, N, K = 2304, 2000, 2048
    assert ozlib.plan_data_drains(M, N, K, 7, 8, 8)
    gen = torch.Generator(device=dev).manual_seed(10)
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
    api.tuning_clear()
    h = ozlib.Handle()
    try:
        h.autotune(M, N, K, 7, 8, 8, max_candidates=1)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
            call(h)
    finally:
        api.tuning_clear()
    dC.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(dC, ref)
    h.close()
