"""Host side of `SplitLinear` without a GPU: what the native description of a forward names.  The library is replaced by a
stand-in that records the descriptions; tensors live on the CPU and only claim to be CUDA tensors."""
import dataclasses

import pytest
import torch

from tailquant_kernel_b200 import _lib, ops
from tailquant_kernel_b200.linear import SplitLinear

FORWARD, PROLOGUE, COMPUTE = "tq_linear_forward", "tq_linear_prologue", "tq_linear_compute"


class Claimed(torch.Tensor):
    """A CPU tensor that passes for a CUDA one (views and copies of it too)."""
    is_cuda = property(lambda self: True)


def claimed(*shape, dtype):
    return torch.zeros(*shape, dtype=dtype).as_subclass(Claimed)


class FakeLibrary:
    def __init__(self, real):
        self.real, self.calls, self.capture = real, [], 0

    def __getattr__(self, name):
        if name == "tq_stream_capture_id":
            return lambda stream: self.capture
        if name not in (FORWARD, PROLOGUE, COMPUTE):
            return getattr(self.real, name)

        def record(call, *rest):
            c = call._obj
            self.calls.append((name, {f: getattr(c, f) for f, _ in c._fields_}))
            return 0
        return record


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary(_lib.load())
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return lib


def weight(N, K, bias=True):
    kind = ops.default_had_kind(K)
    return ops.PreparedWeight(N, K, kind, claimed(N, K // 2, dtype=torch.uint8), claimed(N, dtype=torch.float32),
                              claimed(K, N, dtype=torch.bfloat16), None, claimed(N, K, dtype=torch.bfloat16),
                              claimed(N, dtype=torch.float32) if bias else None)


def layer(N=256, K=512, **kw):
    kw.setdefault("rms_weight", claimed(K, dtype=torch.bfloat16))
    return SplitLinear.from_prepared(weight(N, K), **kw)


def _replace(lin, what):
    if what == "rms_weight":
        lin.rms_weight = claimed(lin.K, dtype=torch.bfloat16)
    elif what == "w":
        lin.w = weight(lin.N, lin.K)
    elif what == "storage":   # as `.to()` or an offloader moves it: the tensor object stays, its memory does not
        lin.w.bias.data = torch.ones(lin.N)
    elif what == "rms_eps":
        lin.rms_eps = 0.25
    else:
        setattr(lin.w, what, torch.clone(getattr(lin.w, what)).as_subclass(Claimed))


@pytest.mark.parametrize("what", ["rms_weight", "bias", "b_col", "w_scale", "w_rot", "w_t", "w", "storage", "rms_eps"])
@pytest.mark.parametrize("M,engine", [(1, "mma"), (20, "mma"), (300, "mma"), (70, "gather")])
def test_a_replaced_part_is_used_by_the_next_call(fake, what, M, engine):
    """No call reads the memory of a weight, bias or norm that the layer no longer holds."""
    lin = layer(tail_engine=engine)
    x = claimed(M, lin.K, dtype=torch.bfloat16)
    for run in (lambda: lin(x), lambda: lin.prologue(x), lambda: lin.compute(lin.workspace(M), M)):
        run()
        _replace(lin, what)
        run()
        c = fake.calls[-1][1]
        w = lin.w
        for field, t in (("b_col", w.b_col), ("w_scale", w.w_scale), ("w_rot", w.w_rot), ("w_t", w.w_t), ("bias", w.bias),
                         ("rms_weight", lin.rms_weight)):
            assert c[field] == t.data_ptr(), field
        assert c["rms_eps"] == lin.rms_eps or what != "rms_eps"


@pytest.mark.parametrize("M,engine,what,bad", [
    (1, "mma", "rms_weight", torch.zeros(512, dtype=torch.bfloat16)),   # on the CPU
    (300, "mma", "rms_weight", claimed(512, dtype=torch.float32)),
    (300, "mma", "rms_weight", claimed(256, dtype=torch.bfloat16)),
    (1, "mma", "bias", claimed(256, dtype=torch.float64)),
    (1, "mma", "bias", claimed(128, dtype=torch.float32)),
    (300, "mma", "w_rot", claimed(256, 256, dtype=torch.bfloat16)),
    (300, "mma", "w_rot", claimed(512, 256, dtype=torch.bfloat16).t()),
    (1, "mma", "w_t", claimed(256, 512, dtype=torch.bfloat16)),
    (70, "gather", "w_t", claimed(512, 256, dtype=torch.float16)),
    (70, "gather", "b_col", claimed(256, 128, dtype=torch.uint8)),
    (70, "gather", "w_scale", claimed(128, dtype=torch.float32))])
def test_a_part_of_the_wrong_kind_is_refused(fake, M, engine, what, bad):
    """Wrong device, type, layout or size: an error, and no native call, from the first forward and from a later one."""
    x = claimed(M, 512, dtype=torch.bfloat16)
    first, later = layer(tail_engine=engine), layer(tail_engine=engine)
    later(x)
    fake.calls.clear()
    for lin in (first, later):
        setattr(lin if what == "rms_weight" else lin.w, what, bad)
        for _ in range(2):
            with pytest.raises(RuntimeError, match=what):
                lin(x)
    assert not fake.calls


def test_an_output_of_the_wrong_kind_is_refused(fake):
    lin = layer()
    ws = lin.prologue(claimed(9, 512, dtype=torch.bfloat16))
    fake.calls.clear()
    for out in (claimed(9, 255, dtype=torch.bfloat16), claimed(9, 256, dtype=torch.float32), torch.zeros(9, 256, dtype=torch.bfloat16)):
        with pytest.raises(RuntimeError, match="out"):
            lin.compute(ws, 9, out)
    assert not fake.calls


def _held(pro):
    bits = {_lib.TQ_OUT_PACK: [pro.a_pack], _lib.TQ_OUT_Q8: [pro.a_q8], _lib.TQ_OUT_LISTS: [pro.tail_idx, pro.tail_val],
            _lib.TQ_OUT_RECORDS: [pro.tail_ptr, pro.tail_rec, pro.tail_cnt], _lib.TQ_OUT_DENSE: [pro.tail_dense]}
    for b, ts in bits.items():
        assert len({t is None for t in ts}) == 1, b
    return sum(b for b, ts in bits.items() if ts[0] is not None)


def _asked(M, N, K, R, kind, engine, shared, sparse=False):
    """`sparse`: beside the 2:4-sparse form of the tail."""
    import ctypes
    call = _lib.LinearCall(M=M, N=N, K=K, R=R, had_kind=kind, engine=engine, sp_val=1 if sparse else None)
    return _lib.load().tq_linear_outputs(ctypes.byref(call), shared)


@pytest.mark.parametrize("R", [0, 26])
@pytest.mark.parametrize("kind,K", [(1, 512), (3, 2048)])
@pytest.mark.parametrize("M", [0, 1, 8, 33, 64, 65, 300, 1024, 1025, 1100, 4096, 4097, 9000])
def test_buffers_of_a_prologue_serve_every_width(M, kind, K, R):
    """Whichever kernel a linear on shared prologue outputs would take on its own, it finds that kernel's operands, or (the
    zero-filled matrix of many rows, kept by narrow layers only) those of the other fused kernel."""
    fused, decode = _lib.TQ_LINEAR_FUSED, _lib.TQ_LINEAR_DECODE
    for n in (8, 136, 1024, 28672):
        held = [_asked(M, n, K, R, kind, e, 1) for e in ((fused, decode) if M <= 64 else (fused,))]
        for h in held:
            for other in (8, 136, 1024, 28672):
                need = _asked(M, other, K, R, kind, fused, 0)
                if M > 1024 and R:
                    need = need & ~_lib.TQ_OUT_DENSE | (need & _lib.TQ_OUT_DENSE and _lib.TQ_OUT_LISTS | _lib.TQ_OUT_RECORDS)
                assert need & ~h == 0, (n, other)
                if M <= 64:
                    assert _asked(M, other, K, R, kind, decode, 0) & ~h == 0
            if kind == 3 and R:
                assert h & _lib.TQ_OUT_DENSE   # long runs of the block rotation


@pytest.mark.parametrize("mode", [-1, 0, 1])
@pytest.mark.parametrize("M", [1, 20, 64, 100, 1000, 1500, 5000])
def test_workspaces_hold_what_the_library_asks_for(fake, M, mode):
    ops.set_gemm_pair_mode(mode)
    try:
        for lin in (layer(), layer(N=24576, K=512, rms_weight=None), layer(ratio=0.0), layer(K=2048), layer(tail_engine="gather")):
            ws = lin.workspace(M)
            assert _held(ws.pro) == _asked(M, lin.N, lin.K, lin.R, lin.w.had_kind, ws.engine, int(lin.tail_engine == "mma"),
                                           ws.pro.sparse is not None)
    finally:
        ops.set_gemm_pair_mode(-1)


@pytest.mark.parametrize("M", [1, 20, 64, 200, 1000, 1500])
def test_a_forward_allocates_what_it_reads(fake, M):
    """No operand of a kernel or a format that the call does not take; what a shared prologue needs beside it comes with the
    first one, and leaves the buffers that a captured graph may name where they are."""
    for lin in (layer(), layer(N=24576, K=512, rms_weight=None), layer(ratio=0.0), layer(K=2048), layer(tail_engine="gather")):
        x = claimed(M, lin.K, dtype=torch.bfloat16)
        lin(x)
        ws = lin._ws[M]
        assert _held(ws.pro) == _asked(M, lin.N, lin.K, lin.R, lin.w.had_kind, ws.engine, 0, ws.pro.sparse is not None)
        before = {f.name: getattr(ws.pro, f.name) for f in dataclasses.fields(ws.pro)}
        assert lin.prologue(x) is ws
        assert _held(ws.pro) == _asked(M, lin.N, lin.K, lin.R, lin.w.had_kind, ws.engine, int(lin.tail_engine == "mma"),
                                       ws.pro.sparse is not None)
        assert all(v is None or getattr(ws.pro, n) is v for n, v in before.items())
        name, c = fake.calls[-1]
        assert name == PROLOGUE and c["a_q8"] == (ws.pro.a_q8.data_ptr() if ws.pro.a_q8 is not None else None)
        assert c["tail_dense"] == (ws.pro.tail_dense.data_ptr() if ws.pro.tail_dense is not None else None)
        lin(x)
        assert lin._ws[M] is ws and _held(ws.pro) == ws.outputs


def test_a_forced_kernel_finds_its_operands(fake):
    lin = layer()
    x = claimed(300, lin.K, dtype=torch.bfloat16)
    lin(x)
    assert not lin._ws[300].outputs & _lib.TQ_OUT_RECORDS
    ops.set_gemm_pair_mode(1)
    try:
        lin(x)
    finally:
        ops.set_gemm_pair_mode(-1)
    assert lin._ws[300].outputs & _lib.TQ_OUT_RECORDS and fake.calls[-1][1]["tail_rec"]


def test_what_a_forward_alone_reads():
    """One format of the codes, and the tail in the one form that the kernel of this shape reads."""
    P, Q, L, T, D = _lib.TQ_OUT_PACK, _lib.TQ_OUT_Q8, _lib.TQ_OUT_LISTS, _lib.TQ_OUT_RECORDS, _lib.TQ_OUT_DENSE
    decode, fused, gather = _lib.TQ_LINEAR_DECODE, _lib.TQ_LINEAR_FUSED, _lib.TQ_LINEAR_GATHER
    assert _asked(4, 4096, 4096, 205, 1, decode, 0) == P | L
    assert _asked(4, 4096, 4096, 0, 1, decode, 0) == P
    assert _asked(300, 4096, 4096, 205, 1, gather, 0) == P | L
    assert _asked(40, 4096, 4096, 205, 1, fused, 0) == Q | D       # 128-channel tiles
    assert _asked(1000, 28672, 4096, 205, 1, fused, 0) == Q | L | T   # CTA pairs
    assert _asked(1000, 28672, 14336, 717, 3, fused, 0) == Q | L | T | D
    assert _asked(1000, 28672, 4096, 0, 1, fused, 0) == Q
    assert _asked(1200, 1200, 14336, 717, 1, fused, 0) == Q | D
    assert _asked(9000, 136, 4096, 205, 1, fused, 0) == Q | L | T
    assert _asked(4, 4096, 4096, 4096, 1, fused, 0) == -1 and _asked(4, 4096, 4096, 5, 1, 3, 0) == -1


@pytest.mark.parametrize("K", [1024, 4096, 12288, 14336])
@pytest.mark.parametrize("ratio", [0.0, 0.01, 0.05, 0.1, 0.4])
def test_one_line_between_decode_and_fused(K, ratio):
    """With more rows a layer goes from the decode kernel over the decode kernel with the tails apart to the fused kernel, and
    never back; rows beyond the single kernel's eight always have the scratch for the tail sums."""
    for N in (8, 256, 1024, 4096, 6144, 12288, 24576, 28672, 65536):
        lin = SplitLinear.__new__(SplitLinear)
        lin.N, lin.K, lin.R, lin.small_m, lin.tail_engine = N, K, ops.ceil_ratio_count(K, ratio), 64, "mma"
        steps = [2 if lin._use_mma(M) else int(lin.R > 0 and lin._tail_apart(M)) for M in range(1, 70)]
        assert steps == sorted(steps), (N, steps)
        assert steps[-1] == 2
        lin.tail_engine = "gather"
        assert not any(lin._use_mma(M) for M in range(1, 70))
        if lin.R:
            assert all(lin._tail_apart(M) for M in range(9, 65))


@pytest.mark.parametrize("N,M,apart", [(24576, 8, True), (24576, 1, False), (256, 4, False), (256, 9, True)])
def test_the_scratch_for_tail_sums_says_where_they_are_made(fake, N, M, apart):
    lin = layer(N=N, K=4096, rms_weight=None, tail_engine="gather")   # (its few rows take the decode engine)
    lin(claimed(M, 4096, dtype=torch.bfloat16))
    c = fake.calls[-1][1]
    assert c["engine"] == _lib.TQ_LINEAR_DECODE and (c["tail"] is not None) == apart


@pytest.fixture
def adapter(fake, monkeypatch):
    """`split_linear_forward` on two prepared layers, reporting which layers ran a prologue."""
    from tailquant_kernel_b200 import linear
    layers, ran = {}, []
    monkeypatch.setattr(linear, "_cached_layer", lambda w, b, r: layers[id(w)])
    monkeypatch.setattr(ops, "_check_cuda", lambda *a, **k: None)
    weights = [claimed(n, 512, dtype=torch.bfloat16) for n in (256, 128)]
    for w in weights:
        lin = layers[id(w)] = layer(N=w.shape[0], rms_weight=None)
        lin.prologue = lambda x, lin=lin: ran.append(lin.N) or SplitLinear.prologue(lin, x)
    linear.clear_cache()

    def call(x, i):
        ran.clear()
        linear.split_linear_forward(x, weights[i])
        return list(ran)
    yield call
    linear.clear_cache()


def test_a_shared_prologue_ends_with_the_next_one(adapter):
    """An input that has to be converted runs a prologue of its own in the layer's buffers: what an earlier input left there
    must not be taken for its prologue any more."""
    x, other = claimed(100, 512, dtype=torch.bfloat16), claimed(100, 512, dtype=torch.float32)
    assert adapter(x, 0) == [256] and adapter(x, 1) == []
    assert adapter(other, 0) == [256]
    assert adapter(x, 1) == [128]
    assert adapter(x, 0) == []


def test_a_capture_contains_the_prologue_of_its_linears(adapter, fake):
    """A replay must not run on what was left by a prologue outside of the graph, nor eager work on a captured one."""
    x = claimed(100, 512, dtype=torch.bfloat16)
    assert adapter(x, 0) == [256] and adapter(x, 1) == []
    for fake.capture in (7, 8, 0):
        assert adapter(x, 0) == [256] and adapter(x, 1) == []


def test_inputs_made_in_inference_mode(adapter):
    """Their in-place changes are not counted: every layer runs its own prologue on them."""
    with torch.inference_mode():
        x = claimed(100, 512, dtype=torch.bfloat16)
        assert adapter(x, 0) == [256] and adapter(x, 1) == [128]
