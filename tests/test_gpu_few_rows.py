"""The kernels for few and medium row counts at the sizes where they can go wrong: edges of row and channel tiles, K ranges
that do not divide, entries beyond a buffer, layers that share a prologue but not a kernel.  Against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

ops = None


@pytest.fixture(scope="module", autouse=True)
def _load():
    global ops
    from tailquant_kernel_b200 import ops as _ops
    ops = _ops
    import test_gpu_parity
    test_gpu_parity.ops = _ops
    yield
    assert ops.gemm_status() == 0, "a bounded device-side wait ran out"


def dev(bits):
    return torch.from_numpy(bits.view(np.int16).copy()).cuda().view(torch.bfloat16)


def host(t):
    return t.detach().contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("M,N,K,R", [(16, 128, 256, 13), (17, 136, 512, 26), (64, 1032, 4096, 205), (65, 264, 1024, 0),
                                     (112, 4096, 512, 60), (176, 256, 4096, 205), (177, 264, 2048, 1), (300, 520, 14336, 717),
                                     (61, 4096, 12288, 615), (353, 128, 1152, 40), (1, 8, 128, 5), (241, 136, 4096, 0), (256, 264, 384, 0),
                                     (1000, 4096, 512, 0)])
def test_shared_k_range_gemm(M, N, K, R):
    """128-channel tiles with the K range of a tile shared by a cluster: accumulators exact, tail sums and outputs inside
    the bounds, at row counts around the 16-row steps and the 176-row tile."""
    from test_gpu_parity import _run_split_gemm_mma
    _run_split_gemm_mma(M, N, K, R, bias=True, cluster=False, pair=0, dense=True)


@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K,kind,ratio", [(1000, 512, O.HAD_WHT, 0.05), (136, 12288, O.HAD_KRON12, 0.05),
                                            (72, 4096, O.HAD_WHT, 0.4), (264, 2048, O.HAD_BLOCK128, 0.0)])
def test_decode_linear_exact(M, N, K, kind, ratio):
    """The one-launch decode linear: bf16 bits of the eight-chain order, ragged channel tiles, few and many tail entries."""
    from tailquant_kernel_b200 import SplitLinear
    xb = O.make_activations(M, K, seed=M, n_outlier=max(1, K // 256))
    wb = O.make_weights(N, K, seed=N)
    b = np.random.default_rng(3).standard_normal(N, dtype=np.float32)
    R = O.ceil_ratio_count(K, ratio)
    ref = O.split_linear_t16(xb, O.prepare_weight(wb, kind), kind, R, bias=b, tail_chains=8)[0]
    lin = SplitLinear(dev(wb), torch.from_numpy(b).cuda(), ratio=ratio, had_kind=kind)
    lin._use_mma = lambda M: False   # this kernel also where the fused one is faster
    for _ in range(2):
        assert np.array_equal(host(lin(dev(xb))), ref)


@pytest.mark.parametrize("M,N,K,ratio,act", [(1, 1000, 512, 0.05, False), (2, 48, 4096, 0.05, True), (5, 72, 4096, 0.4, False),
                                             (8, 272, 2048, 0.01, True), (8, 2056, 1024, 0.002, False),
                                             (2, 16, 14336, 0.6, False)])   # more entries than the tail kernel takes
def test_decode_tail_sums_apart_or_not(M, N, K, ratio, act):
    """Up to eight rows the tail sums come from the decode kernel or from their own: the bits of the eight-chain order."""
    from tailquant_kernel_b200 import SplitLinear
    kind = O.HAD_WHT if K <= 8192 else O.HAD_BLOCK128
    xb, wb = O.make_activations(M, K, seed=M, n_outlier=2), O.make_weights(N, K, seed=N)
    b = np.random.default_rng(3).standard_normal(N, dtype=np.float32)
    got = []
    for apart in (True, False):
        lin = SplitLinear(dev(wb), torch.from_numpy(b).cuda(), ratio=ratio, had_kind=kind, epilogue="swiglu" if act else "none")
        lin._use_mma, lin._tail_apart = lambda M: False, lambda M: apart
        got.append(host(lin(dev(xb))))
        assert (lin._ws[M].tail is not None) == apart
    assert np.array_equal(got[0], got[1])
    if not act:
        R = O.ceil_ratio_count(K, ratio)
        assert np.array_equal(got[0], O.split_linear_t16(xb, O.prepare_weight(wb, kind), kind, R, bias=b, tail_chains=8)[0])


@pytest.mark.parametrize("M,N", [(1, 2056), (2, 6152), (3, 2056), (8, 2056), (40, 2056), (1100, 136)])
def test_few_rows_on_wider_layers(M, N):
    """Widths on which the dispatch between the decode and the fused kernels depends on rows x tail entries."""
    from tailquant_kernel_b200 import SplitLinear
    K, ratio = 1024, 0.05
    xb, wb = O.make_activations(M, K, seed=1, n_outlier=4), O.make_weights(N, K, seed=2)
    R = O.ceil_ratio_count(K, ratio)
    yb, y32, _, _ = O.split_linear_t16(xb, O.prepare_weight(wb, O.HAD_WHT), O.HAD_WHT, R, tail_chains=8)
    got = host(SplitLinear(dev(wb), ratio=ratio)(dev(xb)))
    diff = got != yb
    assert diff.mean() < 0.01 and np.abs(O.bf16_bits_to_f32(got[diff]) - y32[diff]).max(initial=0.0) <= 0.04


@pytest.mark.parametrize("M,ratio", [(8, 0.05), (40, 0.01), (430, 0.10), (700, 0.05)])
def test_layers_on_different_kernels_share_a_prologue(M, ratio):
    """A wide and a narrow layer on one prologue (they may run on different kernels, which read different parts of its
    outputs) give the bits of their own forwards."""
    from tailquant_kernel_b200 import SplitLinear
    K = 1024
    x = dev(O.make_activations(M, K, seed=5, n_outlier=4))
    wide, narrow = (SplitLinear(dev(O.make_weights(n, K, seed=n)), ratio=ratio) for n in (8192, 136))
    want = [wide(x).clone(), narrow(x).clone()]
    for first, second, a, b in ((wide, narrow, 0, 1), (narrow, wide, 1, 0)):
        ws = first.prologue(x)
        ya, yb = first.compute(ws, M), second.compute(ws, M)
        assert torch.equal(ya, want[a]) and torch.equal(yb, want[b])


@pytest.mark.parametrize("M,N,K", [(16, 128, 128), (17, 136, 1152), (112, 4096, 640), (176, 264, 4096), (177, 1000, 2048),
                                   (256, 4096, 4096), (353, 72, 384), (1000, 520, 12288), (1024, 6144, 256)])
@pytest.mark.parametrize("fused", [False, True])
def test_packed_matmul_exact(M, N, K, fused):
    """INT4 x INT4 products on the kernel that shares the K range of a tile: odd slice counts, tile edges in rows and
    channels, few slices per CTA; raw accumulators and the dequantised bf16 output, bit for bit."""
    rng = np.random.default_rng(M + N + K)
    qa, qw = (rng.integers(-8, 8, size=(r, K)).astype(np.int8) for r in (M, N))
    acc = O.int_gemm(qa, qw)
    A, B = (torch.from_numpy(O.pack_s4(q)).cuda() for q in (qa, qw))
    if not fused:
        assert np.array_equal(ops.matmul(A, B).cpu().numpy(), acc)
        return
    sx, sw = (rng.uniform(0.001, 0.02, r).astype(np.float32) for r in (M, N))
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    ops.split_gemm_fused(A, torch.from_numpy(sx).cuda(), B, torch.from_numpy(sw).cuda(), out)
    assert np.array_equal(host(out), O.f32_to_bf16_bits(O.dequant(acc, sx, sw)))


@pytest.mark.parametrize("M,N,K,R", [(1, 8, 64, 1), (3, 1032, 512, 16), (2, 72, 512, 17), (5, 136, 4096, 1024), (2, 16, 4096, 1025)])
def test_t4_sparse_sum_exact(M, N, K, R):
    """Sparse INT4 sums around the 16-entry groups and the staged 1024 entries, at the extreme codes; and an output that is
    not 16-byte aligned."""
    rng = np.random.default_rng(R)
    qw = rng.integers(-8, 8, size=(N, K)).astype(np.int8)
    top_q = rng.integers(-8, 8, size=(M, R)).astype(np.int8)
    qw[0], top_q[0] = -8, -8
    qw[-1] = 7
    idx = np.sort(np.argsort(rng.random((M, K)), axis=1)[:, :R], axis=1).astype(np.int32)
    ts, ws = rng.uniform(0.001, 0.02, M).astype(np.float32), rng.uniform(0.001, 0.02, N).astype(np.float32)
    sp = O.sparse_int_t4(top_q, idx, qw).astype(np.float32)
    want = ((sp * ts[:, None]).astype(np.float32) * ws[None, :]).astype(np.float32)
    g = [torch.from_numpy(a).cuda() for a in (top_q, idx, O.pack_s4(np.ascontiguousarray(qw.T)), ts, ws)]
    for shift in (0, 1):
        out = torch.zeros(M * N + shift, dtype=torch.float16, device="cuda")[shift:].view(M, N)
        ops.sparse_top_write(*g, out)
        assert np.array_equal(out.cpu().numpy(), want.astype(np.float16))


@pytest.mark.parametrize("M,N,K", [(257, 264, 128), (512, 512, 384), (1025, 2056, 512), (1100, 6144, 640)])
def test_pair_kernel_without_a_tail(M, N, K):
    """The paired-SM kernel without a tail: one tile or several per pair, fewer and more K slices than the shared epilogue of
    the last tile needs."""
    from test_gpu_parity import _run_split_gemm_mma
    _run_split_gemm_mma(M, N, K, 0, bias=True, cluster=False, pair=1, dense=True)


@pytest.mark.parametrize("M,N,K,R", [(1, 8, 128, 1), (5, 72, 512, 8), (128, 64, 640, 33), (129, 136, 1024, 64), (40, 4096, 4096, 7),
                                     (300, 2056, 1536, 77), (17, 72, 14336, 3), (9, 16, 2048, 1500)])
def test_gather_chunk_and_batch_edges(M, N, K, R):
    """Ascending-order tail sums, bit for bit: one and few weight chunks, a ragged last chunk, batches of eight entries that
    reach beyond the resident chunks, dense rows, several units of rows per CTA."""
    rng = np.random.default_rng(M + K + R)
    idx = np.sort(np.argsort(rng.random((M, K)), axis=1)[:, :R], axis=1).astype(np.int32)
    idx[0] = np.arange(K - R, K)   # one run at the end of K
    idx[-1] = np.arange(R)
    val, w = O.round_bf16(rng.standard_normal((M, R), dtype=np.float32)), O.round_bf16(rng.standard_normal((K, N), dtype=np.float32))
    want = np.zeros((M, N), np.float32)
    for r in range(R):  # fp32 fma: the product of two bf16 is exact in fp64, and so is its sum up to one rounding
        want = (want.astype(np.float64) + val[:, r:r + 1].astype(np.float64) * w[idx[:, r]]).astype(np.float32)
    out = torch.zeros((M, N), device="cuda")
    ops.tail_gather(torch.from_numpy(idx.astype(np.uint16).view(np.int16)).cuda(), dev(O.f32_to_bf16_bits(val)),
                    dev(O.f32_to_bf16_bits(w)), out, R)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("N,K,kind,ratio", [(520, 1024, O.HAD_WHT, 0.05), (72, 2048, O.HAD_BLOCK128, 0.1), (136, 6144, O.HAD_KRON12, 0.01)])
def test_bits_of_a_row_do_not_depend_on_the_others(N, K, kind, ratio):
    """The exact-order engine without the decode kernel: one row alone, in a few and among many, and the oracle's chain."""
    from tailquant_kernel_b200 import SplitLinear
    M = 300
    xb, wb = O.make_activations(M, K, seed=7, n_outlier=4), O.make_weights(N, K, seed=N)
    b = np.random.default_rng(3).standard_normal(N, dtype=np.float32)
    lin = SplitLinear(dev(wb), torch.from_numpy(b).cuda(), ratio=ratio, had_kind=kind, tail_engine="gather", small_m=0)
    x = dev(xb)
    want = lin(x).clone()
    R = O.ceil_ratio_count(K, ratio)
    assert np.array_equal(host(want[:4]), O.split_linear_t16(xb[:4], O.prepare_weight(wb, kind), kind, R, bias=b)[0])
    for first, rows in ((0, 1), (299, 1), (1, 3), (0, 16), (17, 47), (3, 64), (100, 65), (20, 130)):
        assert torch.equal(lin(x[first:first + rows]), want[first:first + rows]), rows


def test_adapter_in_two_captures():
    """Two graphs captured one after the other on the same static input: each follows the input on its own."""
    from tailquant_kernel_b200 import linear, split_linear_forward
    M, K = 100, 1024
    x = dev(O.make_activations(M, K, seed=1, n_outlier=4))
    ws = [dev(O.make_weights(n, K, seed=n)) for n in (512, 136)]
    linear.clear_cache()
    inputs = [x.clone(), dev(O.make_activations(M, K, seed=2, n_outlier=4))]
    want = [[split_linear_forward(i, w).clone() for w in ws] for i in inputs]
    side = torch.cuda.Stream()
    graphs, outs = [], []
    with torch.cuda.stream(side):
        [split_linear_forward(x, w) for w in ws]
    torch.cuda.synchronize()
    for _ in range(2):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=side):
            outs.append([split_linear_forward(x, w) for w in ws])
    for i in (1, 0):
        x.copy_(inputs[i])
        graphs[i].replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs[i], want[i]))
