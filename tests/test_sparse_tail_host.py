"""When a layer takes its tail as a 2:4-sparse operand, and what it holds for it (no GPU; see test_linear_host.py)."""
import copy
import ctypes
import dataclasses
import pickle
import threading
import time

import pytest
import torch

from tailquant_kernel_b200 import SplitLinear, _lib, ops
from test_linear_host import claimed, fake, layer, weight  # noqa: F401


def sparse(M, N, K, R, kind=1, engine=_lib.TQ_LINEAR_FUSED, shared=0):
    c = _lib.LinearCall(M=M, N=N, K=K, R=R, had_kind=kind, engine=engine)
    return _lib.load().tq_linear_sparse(ctypes.byref(c), shared)


def test_rule():
    assert sparse(2048, 4096, 4096, 205) == 1 and sparse(2048, 4096, 12288, 615, kind=2) == 1
    assert sparse(2048, 4096, 4096, 410) == 0                                 # many entries: groups hold more than two
    assert sparse(2048, 4096, 14336, 717, kind=3) == sparse(2048, 4096, 4096, 205, kind=0) == 0   # not spread over K
    assert sparse(2048, 4096, 4096, 0) == 0 and sparse(2048, 4096, 4096, 205, engine=_lib.TQ_LINEAR_GATHER) == 0
    assert sparse(40, 4096, 4096, 205) == 0 and sparse(300, 1024, 4096, 205) == 0                  # the kernel for few rows
    ops.set_gemm_pair_mode(1)
    try:
        assert sparse(2048, 4096, 4096, 205) == 0
    finally:
        ops.set_gemm_pair_mode(-1)
    assert sparse(2048, 4096, 4096, 4096) == -1


@pytest.mark.parametrize("M", [300, 777, 1500])
def test_a_linear_of_another_width_on_the_same_prologue(fake, M):  # noqa: F811
    """Whichever layer runs the prologue, the others find the operand that they take on their own."""
    lins = [layer(N=n, K=4096, rms_weight=None) for n in (24576, 1024, 4096)]
    for first in lins:
        ws = first.prologue(claimed(M, 4096, dtype=torch.bfloat16))
        assert ws.pro.sparse is not None and (ws.pro.tail_dense is not None or M > 1024)
        for lin in lins:
            lin.w.w_t = None
            lin.compute(ws, M)
            c = fake.calls[-1][1]
            assert c["sp_val"] == ws.pro.sparse[0].data_ptr()
            assert bool(c["w_t"]) == (sparse(M, lin.N, 4096, lin.R) == 1)


@pytest.mark.parametrize("M", [64, 300, 1500])
def test_a_layer_holds_and_names_the_sparse_operand(fake, M):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin(claimed(M, 512, dtype=torch.bfloat16))
    pro, c = lin._ws[M].pro, fake.calls[-1][1]
    if not sparse(M, 24576, 512, lin.R, kind=lin.w.had_kind):
        assert pro.sparse is None and not c["sp_val"]
        return
    assert [t.data_ptr() for t in pro.sparse] == [c[f] for f in ("sp_val", "sp_meta", "sp_over_cnt", "sp_over")]
    assert c["sp_over_ld"] >= (lin.R + 1) // 2 and c["w_t"]


@pytest.mark.parametrize("change", ["replaced", "in_place", "both"])
def test_the_layers_own_transpose_follows_w_rot(fake, change):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    first = lin.w.w_t
    lin(x)
    assert first is not None and lin.w.w_t is first
    if change == "in_place":
        lin.w.w_rot.fill_(2.0)
    else:
        lin.w.w_rot = torch.full_like(lin.w.w_rot, 2.0)
    if change == "both":
        lin.w.w_t = mine = torch.full_like(first, 2.0)
    lin(x)
    assert float(lin.w.w_t[3, 5]) == 2.0 and fake.calls[-1][1]["w_t"] == lin.w.w_t.data_ptr()
    assert change != "both" or lin.w.w_t is mine


def test_a_transpose_is_refreshed_where_it_is(fake):  # noqa: F811
    """A graph captured before still names it."""
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    first, at = lin.w.w_t, lin.w.w_t.data_ptr()
    lin.w.w_rot.fill_(2.0)
    lin(x)
    assert lin.w.w_t is first and lin.w.w_t.data_ptr() == at and float(first[3, 5]) == 2.0


def test_a_transpose_follows_data_put_under_w_rot(fake):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    lin.w.w_rot.data = torch.full_like(lin.w.w_rot, 2.0)
    lin(x)
    assert float(lin.w.w_t[3, 5]) == 2.0


@pytest.mark.parametrize("bad", [claimed(512, 24576, dtype=torch.float16), claimed(24576, 512, dtype=torch.bfloat16),
                                 claimed(24576, 512, dtype=torch.bfloat16).t(), torch.zeros(512, 24576, dtype=torch.bfloat16)])
def test_a_transpose_of_the_wrong_kind_is_refused(fake, bad):  # noqa: F811
    x = claimed(1500, 512, dtype=torch.bfloat16)
    first, later = layer(N=24576, K=512, rms_weight=None), layer(N=24576, K=512, rms_weight=None)
    later(x)
    fake.calls.clear()
    for lin in (first, later):
        lin.w.w_t = bad
        for _ in range(2):
            with pytest.raises(RuntimeError, match="w_t"):
                lin(x)
    assert not fake.calls


def test_a_layer_without_w_rot_is_refused(fake):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_rot = None
    with pytest.raises(RuntimeError):
        lin(claimed(1500, 512, dtype=torch.bfloat16))
    assert not fake.calls


@pytest.mark.parametrize("norm", [False, True])
def test_a_prologue_into_a_workspace_fills_its_sparse_operand(fake, norm):  # noqa: F811
    """The linears on it prefer that operand: one that the prologue left out would be an earlier input's."""
    lin = layer(N=24576, K=512, rms_weight=None)
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    pro = lin.workspace(1500).pro
    assert pro.sparse is not None
    fake.calls.clear()
    gamma = claimed(512, dtype=torch.bfloat16) if norm else None
    assert ops.split_prologue(x, lin.w.had_kind, lin.R, lin.descending_rank, out=pro, rms_weight=gamma) is pro
    (name, c), = fake.calls
    assert name == "tq_linear_prologue" and [t.data_ptr() for t in pro.sparse] == [c[f] for f in ops.SPARSE_FIELDS]
    assert c["a_q8"] == pro.a_q8.data_ptr() and c["rms_weight"] == (gamma.data_ptr() if norm else None)
    assert c["sp_over_ld"] == pro.sparse[3].shape[1]


def test_a_sparse_operand_of_another_size_is_refused(fake):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin(claimed(1500, 512, dtype=torch.bfloat16))
    fake.calls.clear()
    with pytest.raises(RuntimeError, match="sparse"):
        ops.split_prologue(claimed(900, 512, dtype=torch.bfloat16), lin.w.had_kind, lin.R, lin.descending_rank,
                           out=lin.workspace(1500).pro)
    assert not fake.calls


def named(c, pro):
    """The outputs of `pro` that the call `c` names, and those it does not."""
    fields = dict(a_pack="a_pack", a_q8="a_q8", tail_idx="tail_idx16", tail_val="tail_val", tail_ptr="tail_ptr",
                  tail_rec="tail_rec", tail_cnt="tail_cnt", tail_dense="tail_dense")
    pairs = [(getattr(pro, f), c[g]) for f, g in fields.items()] + list(zip(pro.sparse or (), (c[f] for f in ops.SPARSE_FIELDS)))
    return all((t.data_ptr() if t is not None else None) == at for t, at in pairs) and (pro.sparse or not c["sp_val"])


@pytest.mark.parametrize("M", [1, 40, 200, 1000, 1500, 5000])
@pytest.mark.parametrize("N,K", [(24576, 512), (256, 512), (1024, 4096), (256, 2048)])
def test_what_a_workspace_shows_is_what_the_last_call_filled(fake, M, N, K):  # noqa: F811
    """A kernel takes its operand by what it finds: nothing of another call may be among it."""
    lin = layer(N=N, K=K, rms_weight=None)
    x = claimed(M, K, dtype=torch.bfloat16)
    shown = {}
    for run in ("forward", "prologue", "forward", "prologue", "split_prologue"):
        if run == "split_prologue":
            if lin._ws[M].pro.sparse is None:
                continue   # (its entry point takes the outputs one by one)
            ops.split_prologue(x, lin.w.had_kind, lin.R, lin.descending_rank, out=lin.workspace(M).pro)
        else:
            getattr(lin, run)(x)
        pro = lin._ws[M].pro
        assert named(fake.calls[-1][1], pro), run
        assert shown.setdefault(run, pro) is pro
    assert lin._ws[M].held.a_q8 is lin._ws[M].pro.a_q8


def test_a_forward_on_the_sparse_form_holds_no_other_operand(fake):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin(claimed(1500, 512, dtype=torch.bfloat16))
    held = lin._ws[1500].held
    assert held.sparse is not None and held.tail_rec is None and held.tail_cnt is None and held.tail_dense is None


def test_records_are_left_out_where_the_other_forms_are_there(fake):  # noqa: F811
    """Up to 1024 rows a shared prologue leaves the sparse form and the zero-filled matrix; beyond, records and not the matrix."""
    lin = layer(N=24576, K=512, rms_weight=None)
    few, many = lin.workspace(1000).pro, lin.workspace(1500).pro
    assert few.sparse is not None and few.tail_dense is not None and few.tail_rec is None
    assert many.sparse is not None and many.tail_dense is None and many.tail_rec is not None


def test_a_capture_makes_no_transpose(fake):  # noqa: F811
    """It would be written by no kernel before the first replay: the captured forward takes the CTA pairs, later ones make it."""
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    x = claimed(1500, 512, dtype=torch.bfloat16)
    fake.capture = 7
    for _ in range(2):
        lin(x)
        c = fake.calls[-1][1]
        assert c["tail_rec"] and not c["sp_val"] and not c["w_t"] and lin.w.w_t is None
    lin.prepare_decode()
    assert lin.w.w_t is None
    lin.compute(lin.prologue(x), 1500)   # (what several linears read: the sparse form too)
    assert fake.calls[-1][1]["sp_val"] and not fake.calls[-1][1]["w_t"] and lin.w.w_t is None
    fake.capture = 0
    lin(x)
    t = lin.w.w_t
    assert t is not None and fake.calls[-1][1]["sp_val"] and fake.calls[-1][1]["w_t"] == t.data_ptr()
    fake.capture = 8
    lin(x)
    assert fake.calls[-1][1]["w_t"] == t.data_ptr()
    lin.w.w_rot.fill_(2.0)
    lin(x)
    assert not fake.calls[-1][1]["w_t"] and float(t[3, 5]) == 0.0
    fake.capture = 0
    lin(x)
    assert fake.calls[-1][1]["w_t"] == t.data_ptr() and lin.w.w_t is t and float(t[3, 5]) == 2.0


def test_a_captured_decode_call_keeps_its_transpose_to_itself(fake):  # noqa: F811
    lin = layer(rms_weight=None)
    lin.w.w_t = None
    x = claimed(1, 512, dtype=torch.bfloat16)
    fake.capture = 7
    lin(x)
    assert fake.calls[-1][1]["engine"] == _lib.TQ_LINEAR_DECODE and fake.calls[-1][1]["w_t"] and lin.w.w_t is None
    fake.capture = 0
    lin(x)
    assert lin.w.w_t is not None and fake.calls[-1][1]["w_t"] == lin.w.w_t.data_ptr()


@pytest.mark.parametrize("how", ["in_place", "replaced"])
def test_a_sparse_form_that_is_all_there_is_reads_weights_in_line(fake, how):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    lin(claimed(1500, 512, dtype=torch.bfloat16))
    lin.w.w_rot.fill_(2.0)
    if how == "replaced":
        lin.w.w_rot = torch.full_like(lin.w.w_rot, 2.0)
    ops.set_gemm_pair_mode(1)
    try:
        lin.compute(lin._ws[1500], 1500)
    finally:
        ops.set_gemm_pair_mode(-1)
    assert fake.calls[-1][1]["sp_val"] and not fake.calls[-1][1]["w_t"]


def described(**fields):
    """A call on the sparse kernel at 2048 x N x 4096 whose arrays lie at addresses that are never read here."""
    pointers = ("b_col", "w_scale", "w_rot", "w_t", "a_q8", "body_scale", "top_scale", *ops.SPARSE_FIELDS)
    return _lib.LinearCall(**{**dict(M=2048, N=4096, K=4096, R=205, had_kind=1, descending_rank=206, sp_over_ld=104,
                                     engine=_lib.TQ_LINEAR_FUSED), **{f: 0x10000 for f in pointers}, **fields})


@pytest.mark.parametrize("field", ["sp_val", "sp_meta", "sp_over_cnt", "a_q8", "w_t", "w_rot"])
def test_misaligned_operands_are_refused(field):
    c = described(**{field: 0x10008})
    assert _lib.load().tq_linear_compute(ctypes.byref(c), 0x10000, 0) == -3


@pytest.mark.parametrize("N,act,takes", [(4096, 1, 1), (4104, 0, 1), (4104, 1, 0), (4100, 0, 0)])
def test_swiglu_needs_whole_stores(N, act, takes):
    """16 bytes of SwiGLU outputs are 16 channel pairs: other widths stay on the kernels that store them in halves, and where there
    is nothing but the sparse form they are refused."""
    lib, c = _lib.load(), described(N=N, act=act)
    assert lib.tq_linear_sparse(ctypes.byref(c), 0) == takes
    assert ops.takes_sparse(2048, N, 4096, 205, act=act) == bool(takes)
    bits = lib.tq_linear_outputs(ctypes.byref(c), 0)
    assert bool(bits & _lib.TQ_OUT_RECORDS) == (not takes)
    if not takes:
        assert lib.tq_linear_compute(ctypes.byref(c), 0x10000, 0) == -2


@pytest.mark.parametrize("write", ["data", "inference"])
def test_refresh_after_a_write_that_is_not_counted(fake, write):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin.w.w_t = None
    if write == "inference":
        with torch.inference_mode():
            lin.w.w_rot = claimed(24576, 512, dtype=torch.bfloat16)
    lin.refresh()
    assert lin.w.w_t is None
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    t = lin.w.w_t
    with torch.inference_mode():
        lin.w.w_rot.data.fill_(2.0)
    lin.refresh()
    assert lin.w.w_t is t and float(t[3, 5]) == 2.0
    lin(x)
    assert fake.calls[-1][1]["w_t"] == t.data_ptr()
    fake.capture = 7
    with pytest.raises(RuntimeError, match="capture"):
        lin.refresh()


def test_refresh_of_a_transpose_that_cannot_follow(fake):  # noqa: F811
    """Another matrix under `w_rot`: an error instead of a half-written transpose."""
    lin = layer(N=256, K=512, rms_weight=None)
    lin.w.w_rot = claimed(256, 256, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        lin.refresh()


def test_the_prologue_outputs_of_a_forward_by_themselves(fake):  # noqa: F811
    """What the benchmark times as the prologue is what a forward launches."""
    lin = layer(N=24576, K=512, rms_weight=None)
    x = claimed(1500, 512, dtype=torch.bfloat16)
    lin(x)
    pro = lin._ws[1500].pro
    assert lin.workspace(1500, shared=False).pro is pro
    ops.split_prologue(x, lin.w.had_kind, lin.R, lin.descending_rank, out=pro)
    c = fake.calls[-1][1]
    assert c["sp_val"] and c["a_q8"] and not c["tail_rec"] and not c["tail_dense"] and not c["a_pack"]


def test_counts_that_nothing_wrote_are_zero(fake):  # noqa: F811
    """`compute` on a workspace that no prologue has filled finds no left-over entries."""
    lin = layer(N=24576, K=512, rms_weight=None)
    assert int(lin.workspace(1500).pro.sparse[2].abs().sum()) == 0


@pytest.fixture
def patched(fake, monkeypatch):  # noqa: F811
    """`split_linear_forward` on prepared layers of the given widths, as it would make them; reports the prologues that ran."""
    from tailquant_kernel_b200 import linear
    layers = {}
    monkeypatch.setattr(linear, "_cached_layer", lambda w, b, r: layers[id(w)])
    monkeypatch.setattr(ops, "_check_cuda", lambda *a, **k: None)
    linear.clear_cache()

    def make(*widths, K=512):
        weights = [claimed(n, K, dtype=torch.bfloat16) for n in widths]
        for w in weights:
            layers[id(w)] = layer(N=w.shape[0], K=K, rms_weight=None)
            layers[id(w)].split_widths = [w.shape[0]]

        def call(M):
            x = claimed(M, K, dtype=torch.bfloat16)
            fake.calls.clear()
            for w in weights:
                linear.split_linear_forward(x, w)
            return [(name, c["N"], bool(c["sp_val"])) for name, c in fake.calls], [layers[id(w)] for w in weights]
        return call
    yield make
    linear.clear_cache()


def test_a_split_that_takes_no_sparse_operand_gets_none(patched):
    """777 x {4096, 1024, 1024}: none of them does, whatever a wider layer would."""
    call = patched(4096, 1024, 1024, K=4096)
    for _ in range(2):
        calls, lins = call(777)
        assert [c[0] for c in calls] == ["tq_linear_prologue", *["tq_linear_compute"] * 3] and not any(c[2] for c in calls)
        assert lins[0]._ws[777].held.sparse is None and lins[0]._ws[777].pro.tail_dense is not None
    assert lins[0].workspace(300).pro.sparse is None and lins[1].workspace(777).pro.sparse is None


@pytest.mark.parametrize("widths", [(24576, 24576), (24576, 1024)])
def test_a_split_whose_first_linear_takes_it(patched, widths):
    calls, lins = patched(*widths)(1000)
    assert [c[0] for c in calls] == ["tq_linear_prologue", "tq_linear_compute", "tq_linear_compute"]
    assert lins[0]._ws[1000].pro.sparse is not None and calls[0][2]


def test_a_split_whose_later_linear_takes_it(patched):
    """The prologue runs once more when that width follows for the first time: every pass then has the same operands."""
    call = patched(256, 24576)
    calls, lins = call(300)
    assert [c[0].split("_")[-1] for c in calls] == ["prologue", "compute", "prologue", "compute"]
    assert calls[2][1] == 256 and calls[2][2] and calls[3][2]
    calls, lins = call(300)
    assert [c[0].split("_")[-1] for c in calls] == ["prologue", "compute", "compute"] and all(c[2] for c in calls)
    assert call(300)[1][0].split_widths == [256, 24576]


@pytest.mark.parametrize("how", ["in_place", "replaced"])
@pytest.mark.parametrize("first,later", [(1, 1500), (1500, 1), (1, 1), (0, 1500), (0, 1), (0, 0)])
def test_the_transpose_follows_whichever_call_made_it(fake, first, later, how):  # noqa: F811
    """Rows of the call that makes it and of the one after `w_rot` has changed; 0: prepare_decode()."""
    lin = layer(N=8192, K=1024, rms_weight=None)
    lin.w.w_t = None
    call = lambda M: lin(claimed(M, 1024, dtype=torch.bfloat16)) if M else lin.prepare_decode()  # noqa: E731
    call(first)
    t = lin.w.w_t
    assert t is not None
    if how == "in_place":
        lin.w.w_rot.fill_(2.0)
    else:
        lin.w.w_rot = torch.full_like(lin.w.w_rot, 2.0)
    call(later)
    assert float(lin.w.w_t[3, 5]) == 2.0 and (how == "replaced" or lin.w.w_t is t)
    assert later == 0 or fake.calls[-1][1]["w_t"] == lin.w.w_t.data_ptr()


@pytest.mark.parametrize("M", [1, 200])
def test_the_exact_order_engine_follows_w_rot(fake, M):  # noqa: F811
    w = weight(256, 512)
    w.w_t = None
    lin = SplitLinear.from_prepared(w, tail_engine="gather")
    lin.w.w_rot.fill_(2.0)
    lin(claimed(M, 512, dtype=torch.bfloat16))
    assert float(w.w_t[3, 5]) == 2.0 and fake.calls[-1][1]["w_t"] == w.w_t.data_ptr()


def test_layers_on_one_weight_share_its_transpose(fake):  # noqa: F811
    w = weight(8192, 1024)
    w.w_t = None
    a, b = (SplitLinear.from_prepared(w) for _ in range(2))
    a(claimed(1, 1024, dtype=torch.bfloat16))
    t = w.w_t
    w.w_rot.fill_(2.0)
    b(claimed(1500, 1024, dtype=torch.bfloat16))
    assert w.w_t is t and float(t[3, 5]) == 2.0
    a(claimed(1, 1024, dtype=torch.bfloat16))
    assert fake.calls[-1][1]["w_t"] == t.data_ptr()


def test_a_prepared_weight_can_be_copied():
    """What orders streams is not part of a copy."""
    made = object.__new__(ops.Made)
    rot, t = torch.zeros(8, 64), torch.zeros(64, 8)
    w = ops.PreparedWeight(8, 64, 1, torch.zeros(8, 32), torch.zeros(8), t, None, rot, t_of=(t, rot, 0, rot.data_ptr()), t_made=made)
    for twin in (copy.deepcopy(w), pickle.loads(pickle.dumps(w))):
        assert twin.t_made is None and twin.w_t is not t and twin.t_of[0] is twin.w_t and twin.t_of[1] is twin.w_rot


def test_threads_make_one_transpose(fake, monkeypatch):  # noqa: F811
    """Each would read the other's, made on a stream that it does not wait for."""
    lin = layer(N=8192, K=1024, rms_weight=None)
    lin.w.w_t = None
    made, transposed = [], SplitLinear._transposed

    def slow(self, into=None):
        time.sleep(0.05)
        made.append(transposed(self, into))
        return made[-1]
    monkeypatch.setattr(SplitLinear, "_transposed", slow)
    threads = [threading.Thread(target=lin, args=(claimed(M, 1024, dtype=torch.bfloat16),)) for M in (1, 1500, 700)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1 and {c["w_t"] for _, c in fake.calls} == {made[0].data_ptr()} and len(fake.calls) == 3


@pytest.mark.parametrize("which", range(4))
def test_a_gemm_refuses_a_sparse_operand_of_another_size(fake, which):  # noqa: F811
    lin = layer(N=24576, K=512, rms_weight=None)
    lin(claimed(1500, 512, dtype=torch.bfloat16))
    pro, w = lin._ws[1500].pro, lin.w
    sparse = list(pro.sparse)
    sparse[which] = sparse[which][:-1].clone()
    with pytest.raises(RuntimeError, match="sparse"):
        ops.split_gemm_mma(*(t.as_subclass(type(w.b_col)) for t in (pro.a_q8, pro.body_scale)), w.b_col, w.w_scale,
                           claimed(1500, 24576, dtype=torch.bfloat16), w_rot=w.w_rot, pro=dataclasses.replace(pro, sparse=tuple(sparse)),
                           R=lin.R)
