"""The tail as a 2:4-sparse operand: what the prologue writes, and the GEMM that reads it.  The dense part is exact; a tail sum is
an fp32 tensor-core sum of R products, so it differs from the exact one by at most about R roundings of the partial sums, which
|x| |w| R bounds: 1e-5 of that, as for the other fused kernels."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tailquant_kernel_b200 import _lib, ops

pytestmark = pytest.mark.gpu
KINDS = {O.HAD_WHT: _lib.TQ_HAD_WHT, O.HAD_KRON12: _lib.TQ_HAD_KRON12}


def dev(bits):
    return torch.from_numpy(np.ascontiguousarray(bits).view(np.int16)).cuda().view(torch.bfloat16)


def activations(what, M, K, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K, generator=g)
    if what == "hot":
        x[:, torch.randperm(K, generator=g)[:max(1, K // 256)]] *= 50
    elif what == "few_levels":     # channels of equal size: entries come in whole groups
        x[:, [0, 4, 16, 64]] = 300.0
    elif what == "one_row":        # one row of them, and one that is all ties
        x[M // 2, :] = 0.01 * x[M // 2, :]
        x[M // 2, [0, 4]] = 500.0
        x[M // 3, :] = 0.0
        x[M // 3, 5] = 3.0
    elif what == "zeros":          # rotated rows of zeros, and of one value and zeros
        x[::2] = 0.0
        x[1::2] = 1.0
    return x.to(torch.bfloat16).cuda()


def prologue(x, K, R, wide=False, gamma=None, sparse=True):
    """All tail forms of one prologue call, through the native description (`wide`: of the kernel for 16 elements a thread;
    without `sparse` the others)."""
    M = x.shape[0]
    kind = ops.default_had_kind(K)
    e = lambda *s, t: torch.empty(s, dtype=t, device="cuda")  # noqa: E731
    out = dict(a_q8=e(M, K, t=torch.int8), body_scale=e(M, t=torch.float32), top_scale=e(M, t=torch.float32),
               tail_idx16=e(M, (R + 7) // 8 * 8, t=torch.int16), tail_val=e(M, (R + 7) // 8 * 8, t=torch.bfloat16),
               tail_dense=e(M, K, t=torch.bfloat16), sp_val=e(M, K // 2, t=torch.bfloat16), sp_meta=e(M, K // 32, t=torch.int32),
               sp_over_cnt=e(M, t=torch.int16), sp_over=e(M, (R + 1) // 2, t=torch.int32))
    if not sparse:
        out = {k: v for k, v in out.items() if k not in ops.SPARSE_FIELDS}
    c = _lib.LinearCall(M=M, N=8, K=K, R=R, had_kind=kind, descending_rank=ops.split_select_params(K, R)[1],
                        engine=_lib.TQ_LINEAR_FUSED, eps=ops.EPS, tail_ld=out["tail_idx16"].shape[1],
                        sp_over_ld=(R + 1) // 2,
                        rms_weight=None if gamma is None else gamma.data_ptr(), rms_eps=1e-6, **{k: v.data_ptr() for k, v in out.items()})
    lib = _lib.load()
    lib.tq_set_prologue_mode(0 if wide else -1)
    try:
        _lib.check(lib.tq_linear_prologue(ctypes.byref(c), x.data_ptr(), ops._stream()), "prologue")
    finally:
        lib.tq_set_prologue_mode(-1)
    torch.cuda.synchronize()
    return out


# (what, rows, K, R, kernel): the kernel of 16 elements a thread, or that of 64, which K = 4096 takes beyond 256 rows and K = 12288
# beyond 128 and which can be kept off
CASES = [("plain", 3, 512, 26, 16), ("one_row", 300, 4096, 205, 16), ("few_levels", 130, 4096, 287, 16), ("zeros", 20, 1024, 52, 16),
         ("plain", 9, 2048, 1, 16), ("hot", 20, 12288, 615, 16), ("zeros", 140, 12288, 615, 16), ("one_row", 33, 6144, 400, 16),
         ("few_levels", 40, 8192, 410, 16), ("hot", 300, 4096, 205, 64), ("one_row", 300, 4096, 205, 64),
         ("few_levels", 300, 4096, 287, 64), ("zeros", 300, 4096, 205, 64), ("hot", 140, 12288, 615, 64), ("few_levels", 140, 12288, 860, 64), ("zeros", 140, 12288, 615, 64)]


@pytest.mark.parametrize("what,M,K,R,elements", CASES)
@pytest.mark.parametrize("norm", [False, True])
def test_prologue_writes_the_tail_in_sparse_form(what, M, K, R, elements, norm):
    """The first two entries of each group in order with their places, all others in the row's list; only zeros are left out.
    What else is written has the bits of a prologue without the sparse form (which is compared with the oracle)."""
    gamma = (1 + 0.1 * torch.randn(K, generator=torch.Generator().manual_seed(1))).to(torch.bfloat16).cuda() if norm else None
    x = activations(what, M, K, 11)
    o = prologue(x, K, R, elements == 16, gamma)
    for name, t in prologue(x, K, R, elements == 16, gamma, sparse=False).items():
        mine = o[name]
        if name in ("tail_idx16", "tail_val"):   # (padded to whole stores)
            t, mine = t[:, :R].contiguous(), mine[:, :R].contiguous()
        assert torch.equal(t.view(torch.uint8), mine.view(torch.uint8)), name
    want = o["tail_dense"].view(torch.int16).cpu().numpy().astype(np.int64) & 0xffff
    member = np.zeros((M, K), bool)
    np.put_along_axis(member, o["tail_idx16"].cpu().numpy()[:, :R].astype(np.int64) & 0xffff, True, 1)
    val = (o["sp_val"].view(torch.int16).cpu().numpy().astype(np.int64) & 0xffff).reshape(M, K // 4, 2)
    meta = o["sp_meta"].cpu().numpy().view(np.uint32).astype(np.int64)
    nib = ((meta[:, :, None] >> (4 * np.arange(8))) & 15).reshape(M, K // 4)
    lo, hi = nib & 3, nib >> 2
    assert (lo < hi).all(), "places in order"
    got = np.zeros((M, K // 4, 4), np.int64)
    np.put_along_axis(got, np.stack((lo, hi), -1), val, -1)
    cnt, over = o["sp_over_cnt"].cpu().numpy().astype(np.int64), o["sp_over"].cpu().numpy().view(np.uint32).astype(np.int64)
    assert (cnt >= 0).all() and (cnt <= (R + 1) // 2).all()
    flat = got.reshape(M, K)
    for m in range(M):
        k, v = over[m, :cnt[m]] & 0xffff, over[m, :cnt[m]] >> 16
        assert (np.diff(k) > 0).all()
        nz = (want[m] & 0x7fff) != 0
        tail = member[m] & nz if (want[m][member[m]] & 0x7fff).min() == 0 else member[m]
        rank = np.cumsum(tail.reshape(-1, 4), 1).reshape(-1)
        assert np.array_equal(k, np.flatnonzero(tail & (rank > 2))), "entries beyond two of a group"
        assert (flat[m][k] == 0).all()
        flat[m][k] = v
    assert np.array_equal(flat, want)


@pytest.mark.parametrize("what,M,N,K,ratio", [
    ("plain", 1, 8, 512, 0.05), ("plain", 129, 232, 512, 0.05), ("hot", 257, 456, 1024, 0.05), ("hot", 300, 264, 4096, 0.05),
    ("few_levels", 300, 240, 2048, 0.05), ("one_row", 520, 224, 4096, 0.05), ("zeros", 64, 40, 1024, 0.05),
    ("hot", 200, 72, 12288, 0.05), ("plain", 2000, 4096, 512, 0.07), ("plain", 300, 1000, 6144, 0.001)])
@pytest.mark.parametrize("with_t", [True, False])
def test_gemm_on_the_sparse_tail(what, M, N, K, ratio, with_t):
    """Rows and channels that do not fill a tile, several tiles per pair, many and no left-over entries, with and without the
    transposed weights: accumulators bit for bit, tail sums and outputs inside the bound."""
    R = ops.ceil_ratio_count(K, ratio)
    o = prologue(activations(what, M, K, 5), K, R)
    g = torch.Generator().manual_seed(N)
    w = ops.prepare_weight((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda(), t16=True, keep_w_rot=True)
    bias = torch.randn(N, generator=g).cuda()
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    acc, tail = torch.empty((M, N), dtype=torch.int32, device="cuda"), torch.empty((M, N), device="cuda")
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    _lib.check(_lib.load().tq_split_gemm_sparse(
        p(o["a_q8"]), p(o["body_scale"]), p(w.b_col), p(w.w_scale), p(w.w_rot), p(w.w_t) if with_t else None, R, p(o["sp_val"]),
        p(o["sp_meta"]), p(o["sp_over_cnt"]), p(o["sp_over"]), o["sp_over"].shape[1], p(bias), p(out), p(acc), p(tail), M, N, K, 0,
        ops._stream()), "sparse gemm")
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0
    codes = o["a_q8"].cpu().numpy().reshape(M, K // 8, 8)[:, :, [0, 4, 1, 5, 2, 6, 3, 7]].reshape(M, K).astype(np.float64)
    qw = O.unpack_s4(w.b_col.cpu().numpy()).astype(np.float64)
    assert np.array_equal(acc.cpu().numpy(), (codes @ qw.T).astype(np.int64))
    wr, d = w.w_rot.double(), o["tail_dense"].double()
    exact = (d @ wr.T).cpu().numpy()
    bound = 1e-5 * R * float(d.abs().max()) * float(wr.abs().max())
    assert np.abs(tail.cpu().numpy() - exact).max() <= bound
    y = (acc.float() * o["body_scale"][:, None]) * w.w_scale[None] + tail + bias[None]
    assert torch.equal(out, y.to(torch.bfloat16)), "dequantised, tail and bias added, rounded once"


@pytest.mark.parametrize("M,N,K", [(700, 8192, 1024), (1500, 4096, 4096)])
def test_layer_with_swiglu_on_the_sparse_tail(M, N, K):
    """The layer object takes the sparse operand at this size; SwiGLU in the epilogue against the plain layer's outputs."""
    from tailquant_kernel_b200 import SplitLinear, interleave_gate_up
    x = activations("hot", M, K, 3)
    g = torch.Generator().manual_seed(9)
    wg, wu = ((torch.randn(N // 2, K, generator=g) * 0.02).to(torch.bfloat16).cuda() for _ in range(2))
    W = interleave_gate_up(wg, wu)
    plain, fused = SplitLinear(W), SplitLinear(W, epilogue="swiglu")
    y, h = plain(x), fused(x)
    assert plain._ws[M].pro.sparse is not None and fused._ws[M].pro.sparse is not None
    want = (torch.nn.functional.silu(y[:, 0::2].float()).to(torch.bfloat16).float() * y[:, 1::2].float()).to(torch.bfloat16)
    diff = want.float() - h.float()
    assert (diff != 0).float().mean() < 2e-3 and bool((diff.abs() <= want.float().abs() * 2.0 ** -7 + 1e-30).all())
    ops.set_gemm_pair_mode(1)
    try:
        ref = SplitLinear(W)(x).float()
    finally:
        ops.set_gemm_pair_mode(-1)
    d = (y.float() - ref).abs()
    assert float((d != 0).float().mean()) < 1e-3 and bool((d <= ref.abs() * 2.0 ** -7 + 1e-4).all())


@pytest.mark.parametrize("with_t", [True, False])
def test_outputs_that_no_prologue_filled_are_read_inside_their_arrays(with_t):
    """Counts beyond the list and indices beyond K, as memory that nothing wrote may hold them: the tail is of no use, the dense
    part and the status are in order."""
    M, N, K, R = 300, 264, 512, 26
    o = prologue(activations("plain", M, K, 5), K, R)
    o["sp_over_cnt"].fill_(-1)
    o["sp_over"].copy_(torch.randint(-2 ** 31, 2 ** 31, o["sp_over"].shape, dtype=torch.int64).to(torch.int32).cuda())
    w = ops.prepare_weight((torch.randn(N, K) * 0.02).to(torch.bfloat16).cuda(), t16=True, keep_w_rot=True)
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    acc = torch.empty((M, N), dtype=torch.int32, device="cuda")
    p = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(_lib.load().tq_split_gemm_sparse(
        p(o["a_q8"]), p(o["body_scale"]), p(w.b_col), p(w.w_scale), p(w.w_rot), p(w.w_t) if with_t else None, R,
        *(p(o[f]) for f in ops.SPARSE_FIELDS), o["sp_over"].shape[1], None, p(out), p(acc), None, M, N, K, 0, ops._stream()), "gemm")
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0
    codes = o["a_q8"].cpu().numpy().reshape(M, K // 8, 8)[:, :, [0, 4, 1, 5, 2, 6, 3, 7]].reshape(M, K).astype(np.float64)
    assert np.array_equal(acc.cpu().numpy(), (codes @ O.unpack_s4(w.b_col.cpu().numpy()).astype(np.float64).T).astype(np.int64))


def test_swiglu_of_a_width_that_the_sparse_kernel_does_not_store():
    """N % 16 == 8: the kernel on records, whatever else the prologue left."""
    M, N, K = 1500, 8200, 1024
    x = activations("hot", M, K, 3)
    g = torch.Generator().manual_seed(9)
    w = ops.prepare_weight((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda(), t16=False, keep_w_rot=True)
    from tailquant_kernel_b200 import SplitLinear
    plain = SplitLinear.from_prepared(w)
    y, pro = plain(x).clone(), plain.workspace(M).pro
    assert pro.sparse is not None and ops.takes_sparse(M, N, K, plain.R) and not ops.takes_sparse(M, N, K, plain.R, act=1)
    ops.split_prologue(x, w.had_kind, plain.R, plain.descending_rank, out=pro)
    h = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
    ops.split_gemm_mma(pro.a_q8, pro.body_scale, w.b_col, w.w_scale, h, w_rot=w.w_rot, pro=pro, R=plain.R, act="swiglu")
    gate, up = y[:, 0::2].float(), y[:, 1::2].float()
    silu = torch.nn.functional.silu(gate)
    want = (silu.to(torch.bfloat16).float() * up).to(torch.bfloat16).float()
    # other order of the tail sum: a gate or an up value moves by a last place now and then, 2^-7 of it at most (|silu'| <= 1.1),
    # and silu and the product are rounded again
    bound = 2.0 ** -7 * (1.1 * (gate * up).abs() + 3 * (silu * up).abs()) + 1e-30
    diff = (want - h.float()).abs()
    assert float((diff != 0).float().mean()) < 2e-3 and bool((diff <= bound).all())


def test_weights_changed_in_place_reach_the_left_over_entries():
    """The transposed weights are a copy that the layer made: it follows `w_rot`."""
    from tailquant_kernel_b200 import SplitLinear
    M, N, K = 1100, 4096, 1024
    x = activations("few_levels", M, K, 1)
    g = torch.Generator().manual_seed(2)
    w = (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda()
    lin = SplitLinear(w)
    lin(x)
    assert lin._ws[M].pro.sparse is not None
    other = SplitLinear(2 * w)
    t = lin.w.w_t
    lin.w.w_rot.copy_(other.w.w_rot)
    lin.w.b_col.copy_(other.w.b_col)
    lin.w.w_scale.copy_(other.w.w_scale)
    assert torch.equal(lin(x), other(x)) and lin.w.w_t is t and torch.equal(t, lin.w.w_rot.t())
    lin.w.w_rot = SplitLinear(w).w.w_rot
    other.w.w_rot, other.w.w_t = lin.w.w_rot, None
    assert torch.equal(lin(x), other(x))


@pytest.mark.parametrize("M", [700, 1500])
def test_a_prologue_into_a_used_workspace(M):
    """Another input through `split_prologue`, then the GEMM by either entry point: the outputs of a layer that never saw the first."""
    from tailquant_kernel_b200 import SplitLinear
    N, K = 8192, 1024
    g = torch.Generator().manual_seed(4)
    w = (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda()
    lin, fresh = SplitLinear(w), SplitLinear(w)
    lin(activations("few_levels", M, K, 1))
    assert lin._ws[M].pro.sparse is not None
    x = activations("hot", M, K, 2)
    ws = lin.workspace(M)
    ops.split_prologue(x, lin.w.had_kind, lin.R, lin.descending_rank, out=ws.pro)
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    ops.split_gemm_mma(ws.pro.a_q8, ws.pro.body_scale, lin.w.b_col, lin.w.w_scale, out, w_rot=lin.w.w_rot, pro=ws.pro, R=lin.R)
    y = fresh(x)
    assert torch.equal(out, y) and torch.equal(lin.compute(ws, M), y)


def test_refresh_after_a_write_that_is_not_counted():
    """As a collective into `w_rot` leaves it; a captured graph follows, since the transpose stays where it is."""
    from tailquant_kernel_b200 import SplitLinear
    M, N, K = 1500, 8192, 1024
    g = torch.Generator().manual_seed(7)
    a, b = ((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda() for _ in range(2))
    lin, other = SplitLinear(a), SplitLinear(b)
    x = activations("few_levels", M, K, 2)
    lin(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin(x)
    for f in ("w_rot", "b_col", "w_scale"):
        getattr(lin.w, f).data.copy_(getattr(other.w, f))
    lin.refresh()
    graph.replay()
    assert torch.equal(y, other(x)) and torch.equal(lin(x), other(x))


@pytest.mark.parametrize("M", [1, 700, 1500])
@pytest.mark.parametrize("maker", ["default", "side"])
def test_a_transpose_made_on_another_stream_is_waited_for(M, maker):
    """The call that makes it is held up on its stream; the next one, of another row count, comes on a stream of its own."""
    from tailquant_kernel_b200 import SplitLinear
    N, K = 8192, 1024
    g = torch.Generator().manual_seed(5)
    lin = SplitLinear((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda())
    fresh = SplitLinear.from_prepared(ops.PreparedWeight(**{**vars(lin.w), "w_t": None}))
    x, first = activations("few_levels", M, K, 2), activations("plain", 1000, K, 1)
    want = fresh(x).clone()
    torch.empty((K, N), dtype=torch.bfloat16, device="cuda").fill_(7.0)   # (what the transpose's memory may have held)
    side, default = torch.cuda.Stream(), torch.cuda.current_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side if maker == "side" else default):
        torch.cuda._sleep(20_000_000)   # (some 10 ms)
        lin(first)
    assert lin.w.w_t is not None
    with torch.cuda.stream(default if maker == "side" else side):
        y = lin(x)
        assert torch.equal(y, want)


@pytest.mark.parametrize("M", [1, 1500])
def test_a_capture_that_is_the_first_call_on_the_transposed_weights(M):
    """Eager calls between the capture and its first replay read a transpose of their own; the captured one sums the tail on
    another kernel (a bf16 step apart where a sum lies near the middle)."""
    from tailquant_kernel_b200 import SplitLinear
    N, K = 8192, 1024
    g = torch.Generator().manual_seed(5)
    lin = SplitLinear((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda())
    fresh = SplitLinear.from_prepared(ops.PreparedWeight(**{**vars(lin.w), "w_t": None}))
    lin(activations("plain", 300, K, 1)), torch.cuda.synchronize()
    x, out = activations("few_levels", M, K, 2), []
    lin.w.w_t = None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out.append(lin(x))
    assert lin.w.w_t is None
    want = fresh(x)
    assert torch.equal(lin(x), want) and torch.equal(lin.w.w_t, lin.w.w_rot.t())
    out[0].zero_()
    graph.replay()
    d, want = (out[0].float() - want.float()).abs(), want.float().abs()
    sums = 1e-5 * lin.R * (4 * 300 / K ** 0.5 + 6) * float(lin.w.w_rot.abs().max())   # (a few_levels row's largest rotated value)
    assert float((d != 0).float().mean()) < 1e-3 and bool((d <= want * 2.0 ** -7 + sums).all())


def outputs(pro):
    return [t for t in (pro.a_pack, pro.a_q8, pro.body_scale, pro.tail_idx, pro.tail_val, pro.tail_ptr, pro.tail_rec, pro.tail_cnt,
                        pro.tail_dense, *(pro.sparse or ())) if t is not None]


@pytest.mark.parametrize("M,N,K", [(3, 512, 1024), (40, 512, 1024), (200, 8192, 1024), (1000, 4096, 1024), (1000, 4096, 4096),
                                   (1500, 8192, 1024), (1500, 4096, 2048)])
def test_every_output_shown_is_written(M, N, K):
    """By a forward and by a prologue for several linears, in turn on inputs of their own: whatever a kernel finds there is of
    this input, and the results are those of a fresh layer."""
    from tailquant_kernel_b200 import SplitLinear
    g = torch.Generator().manual_seed(6)
    w = (torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda()
    lin = SplitLinear(w, had_kind=3 if K == 2048 else None)
    for seed, run in enumerate((lin.forward, lin.prologue, lin.forward, lin.prologue)):
        x = activations("few_levels", M, K, seed)
        lin.workspace(M)
        if run == lin.forward:
            lin._workspace(M, False)
        shown = outputs(lin._ws[M].pro)
        for t in shown:
            t.view(torch.uint8).fill_(0x5b)
        run(x)
        assert [t.data_ptr() for t in outputs(lin._ws[M].pro)] == [t.data_ptr() for t in shown]
        for t in shown:
            assert not bool((t.view(torch.uint8) == 0x5b).all())
        y = lin.compute(lin._ws[M], M).clone()
        fresh = SplitLinear.from_prepared(lin.w)
        assert torch.equal(y, fresh(x))


@pytest.mark.parametrize("mode", [0, 1])
def test_another_kernel_after_a_forward_on_the_sparse_form(mode):
    """It finds the sparse form and nothing else of the tail, and takes that."""
    from tailquant_kernel_b200 import SplitLinear
    M, N, K = 1500, 8192, 1024
    g = torch.Generator().manual_seed(8)
    lin = SplitLinear((torch.randn(N, K, generator=g) * 0.02).to(torch.bfloat16).cuda())
    y = lin(activations("hot", M, K, 3)).clone()
    pro = lin._ws[M].pro
    assert pro.sparse is not None
    out = torch.empty_like(y)
    ops.set_gemm_pair_mode(mode)
    try:
        ops.split_gemm_mma(pro.a_q8, pro.body_scale, lin.w.b_col, lin.w.w_scale, out, w_rot=lin.w.w_rot, pro=pro, R=lin.R)
        assert torch.equal(out, y) and torch.equal(lin.compute(lin._ws[M], M), y)
    finally:
        ops.set_gemm_pair_mode(-1)


def test_swiglu_of_every_gate():
    """The epilogues' quotient has the bits of the IEEE division for every bf16 gate, infinities and the largest ones among them
    (NaN where that is NaN); the finisher of the split-K path rounds it to bf16."""
    q, d = torch.empty(65536, device="cuda"), torch.empty(65536, device="cuda")
    _lib.check(_lib.load().tq_swiglu_quotients(q.data_ptr(), d.data_ptr(), ops._stream()), "quotients")
    nan = torch.isnan(d)
    assert torch.equal(torch.isnan(q), nan) and torch.equal(q.view(torch.int32)[~nan], d.view(torch.int32)[~nan])
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).float().cuda()
    n = g.numel()
    y = torch.stack((g, torch.ones_like(g)), 1).reshape(1, -1).contiguous()
    acc, one = torch.zeros((1, 1, 2 * n), dtype=torch.int32, device="cuda"), torch.ones(2 * n, device="cuda")
    out = torch.empty((1, n), dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.load().tq_dequant_finish_partials(acc.data_ptr(), 1, one.data_ptr(), one.data_ptr(), y.data_ptr(), None,
                                                      out.data_ptr(), 1, 2 * n, 1, ops._stream()), "finish")
    assert torch.equal(torch.isnan(out[0]), nan) and torch.equal(out[0][~nan], d[~nan].to(torch.bfloat16))
