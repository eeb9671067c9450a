"""The split W4A4 + tail linear as a host-side object, and the module-level callable the
reference's drop-in adapter discovers.

Forward of one linear (mirrors the step list of `RealPolicyLinear.forward` as restated in
tools/profile_multimodel_split_components_v34.py:93-272):
    prologue (rotation + select + pack)  ->  tail gather (R > 0)  ->  GEMM with fused dequant,
    tail add and bias.  A few rows take the decode kernel instead (see `SplitLinear`).
The kernels of a forward are enqueued by one native call (`tq_linear_forward`) on a description that is filled in once
per row count, and again when a weight, the bias or the norm was replaced.  Everything runs on the current CUDA stream out of per-(M) workspaces that are allocated once, so
a forward is capturable in a CUDA graph after its first call, as the reference's benches require
(tools/bench_hadamard_three_schemes_quarot_dense_sharedqkv_inplace_fusedtopr_v43.py:105-123).
"""
from __future__ import annotations

import ctypes
import threading
import weakref
from collections import OrderedDict
from typing import Dict, List, Optional, Tuple

import torch

from . import _lib, ops


_MAKING = threading.Lock()   # held while a transpose of rotated weights is made


def interleave_gate_up(w_gate: torch.Tensor, w_up: torch.Tensor) -> torch.Tensor:
    """[2 I, K] weight of a fused gate_up projection with rows (gate_0, up_0, gate_1, up_1, ...): the layout
    `SplitLinear(..., epilogue="swiglu")` expects."""
    if w_gate.shape != w_up.shape or w_gate.dim() != 2:
        raise RuntimeError("gate and up weights must be [I, K] tensors of the same shape")
    return torch.stack((w_gate, w_up), dim=1).reshape(2 * w_gate.shape[0], w_gate.shape[1]).contiguous()


class _Workspace:
    """Buffers of one (layer, M): the prologue outputs (absent in the workspace a layer uses when it runs on another layer's
    prologue) and the layer's own output and scratch.  They stay for as long as the layer does and are only ever added to,
    since captured graphs name them: a row count that is seen once costs what its forward reads.  `pro` shows those of the
    prologue outputs that are filled together, by a forward or by a prologue for several linears: a kernel chooses its
    operand by what it finds, and must not find what another call left."""

    def __init__(self, M: int, N: int, K: int, R: int, device, engine: int, n_out: int, with_pro: bool,
                 with_tail: bool):
        empty = lambda shape, dtype: torch.empty(shape, dtype=dtype, device=device)  # noqa: E731
        self.M, self.K, self.R, self.engine = M, K, R, engine
        self.held = None   # all prologue outputs
        self.pro = None    # the ones in use, `outputs` and `sparse` of show()
        self.outputs = 0
        self.forward_for = self.shared_for = -1   # forced-kernel state (see ops) that `pro` was chosen under, -1: not `pro`
        self._views: Dict[Tuple[int, bool], ops.PrologueOut] = {}
        if with_pro:
            self.held = ops.PrologueOut(a_pack=None, body_scale=empty(M, torch.float32), top_scale=empty(M, torch.float32),
                                        tail_idx=None, tail_val=None, R=R)
        self.tail = empty((M, N), torch.float32) if with_tail else None   # sums of a tail kernel of its own
        self.out = empty((M, n_out), torch.bfloat16)
        self.call = None   # (a reference to) the native description of a forward out of these buffers; what it was filled in from
        self.call_pro = None
        self.call_src = ()
        self.call_t = None
        self.rot_version = None   # of w_rot, where the description rests on its transpose

    _FIELDS = {_lib.TQ_OUT_PACK: ("a_pack",), _lib.TQ_OUT_Q8: ("a_q8",), _lib.TQ_OUT_LISTS: ("tail_idx", "tail_val"),
               _lib.TQ_OUT_RECORDS: ("tail_ptr", "tail_rec", "tail_cnt"), _lib.TQ_OUT_DENSE: ("tail_dense",)}

    def show(self, outputs: int, sparse: bool) -> None:
        """Has `pro` be the prologue outputs of `outputs` (TQ_OUT_* bits) and, with `sparse`, the 2:4-sparse form of the tail,
        making those that are not there yet."""
        view = self._views.get((outputs, sparse))
        if view is None:
            self._make(outputs, sparse)
            h = self.held
            view = ops.PrologueOut(a_pack=None, body_scale=h.body_scale, top_scale=h.top_scale, tail_idx=None, tail_val=None,
                                   R=h.R, sparse=h.sparse if sparse else None)
            for bit, names in self._FIELDS.items():
                for name in names if outputs & bit else ():
                    setattr(view, name, getattr(h, name))
            self._views[outputs, sparse] = view
        self.pro, self.outputs = view, outputs

    def _make(self, outputs: int, sparse: bool) -> None:
        p, M, K, R, device = self.held, self.M, self.K, self.R, self.out.device
        empty = lambda shape, dtype: torch.empty(shape, dtype=dtype, device=device)  # noqa: E731
        if outputs & _lib.TQ_OUT_PACK and p.a_pack is None:
            p.a_pack = empty((M, K // 2), torch.uint8)
        if outputs & _lib.TQ_OUT_Q8 and p.a_q8 is None:
            p.a_q8 = empty((M, K), torch.int8)
        if outputs & _lib.TQ_OUT_LISTS and p.tail_idx is None:
            p.tail_idx = torch.zeros((M, (R + 7) // 8 * 8), dtype=torch.int16, device=device)
            p.tail_val = torch.zeros((M, (R + 7) // 8 * 8), dtype=torch.bfloat16, device=device)
        if outputs & _lib.TQ_OUT_RECORDS and p.tail_ptr is None:
            half_slices = (2 * ((M + 255) // 256), K // 64, 128)
            p.tail_ptr = empty((M, K // 128 + 1), torch.int16)
            p.tail_rec = empty((*half_slices, ops.TAIL_REC_CAP), torch.int32)
            p.tail_cnt = torch.zeros(half_slices, dtype=torch.int16, device=device)
        if outputs & _lib.TQ_OUT_DENSE and p.tail_dense is None:
            p.tail_dense = empty((M, K), torch.bfloat16)
        if sparse and p.sparse is None:
            p.sparse = (empty((M, K // 2), torch.bfloat16), empty((M, K // 32), torch.int32),
                        torch.zeros((M,), dtype=torch.int16, device=device), empty((M, (R + 1) // 2), torch.int32))


class SplitLinear:
    """Prepared weights + workspaces of one linear layer y = x W^T (+ bias)."""

    def __init__(self, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, ratio: float = 0.05,
                 activation_percentile: float = 100.0, had_kind: Optional[int] = None, small_m: int = 64,
                 split_k: int = 0, tail_engine: str = "mma", epilogue: str = "none",
                 rms_weight: Optional[torch.Tensor] = None, rms_eps: float = 1e-6, reuse_output: bool = True):
        """tail_engine: "mma" = tail on the tensor cores inside the GEMM kernel (default, fastest at
        ratios of a few percent); a few rows take the decode kernel where that is faster.  The order of a tail sum, and
        with it the last place of an output now and then, then depends on how many rows come together.  "gather" = fp32
        fma chains in a stated order on the CUDA cores, bit-exact against the CPU oracle: one ascending chain per output
        beyond `small_m` rows, eight interleaved ones (the decode kernel's) up to `small_m`.  With small_m=0 the bits of
        a row do not depend on the rows that come with it.
        small_m: rows up to which the decode kernel is considered (at most 64; with the "mma" engine at most 32 count).
        split_k: without effect, kept for existing calls: the integer sums are exact however K is split.
        epilogue: "swiglu" = `weight` is a fused gate_up matrix with interleaved rows (`interleave_gate_up`) and the
        layer returns bf16(bf16(silu(gate)) * up), [.., N/2], without writing the [.., N] intermediate.
        rms_weight: [K] bf16 weight of an RMSNorm that precedes this linear: the layer then takes the UN-normalised
        hidden state and applies the norm inside its prologue kernel.
        reuse_output: True (default) returns the layer's per-M output buffer, which the next forward with the same M
        overwrites -- no allocation per call, what a captured CUDA graph needs; False returns a fresh tensor."""
        if tail_engine not in ("mma", "gather"):
            raise RuntimeError("tail_engine must be 'mma' or 'gather'")
        if epilogue not in ("none", "swiglu"):
            raise RuntimeError("epilogue must be 'none' or 'swiglu'")
        if epilogue == "swiglu" and (tail_engine != "mma" or weight.shape[0] % 16):
            raise RuntimeError("the SwiGLU epilogue needs the 'mma' tail engine and N % 16 == 0")
        if not weight.is_cuda:
            raise RuntimeError("SplitLinear needs CUDA weights: there is no CPU path")
        K = int(weight.shape[1])
        R = ops.ceil_ratio_count(K, float(ratio))
        # the [K, N] transpose of the rotated weights serves the gather engine and the decode tail; with the
        # tensor-core tail it is built by `prepare_decode()` or on the first small-M call (it doubles the bf16
        # weight memory)
        w = ops.prepare_weight(weight, had_kind, t16=R > 0 and tail_engine == "gather",
                               keep_w_rot=R > 0 and tail_engine == "mma", bias=bias)
        self._init(w, ratio, activation_percentile, small_m, split_k, tail_engine, epilogue,
                   None if rms_weight is None else rms_weight.detach().to(torch.bfloat16).contiguous(), rms_eps,
                   reuse_output)

    def _init(self, w: "ops.PreparedWeight", ratio, activation_percentile, small_m, split_k, tail_engine, epilogue,
              rms_weight, rms_eps, reuse_output) -> None:
        self.w = w
        self.N, self.K = int(w.N), int(w.K)
        self.ratio = float(ratio)
        self.R = ops.ceil_ratio_count(self.K, self.ratio)
        self.activation_percentile = float(activation_percentile)
        _, self.descending_rank, _ = ops.split_select_params(self.K, self.R, self.activation_percentile)
        self.small_m, self.split_k = int(small_m), int(split_k)
        self.tail_engine, self.epilogue = tail_engine, epilogue
        self.rms_weight, self.rms_eps = rms_weight, float(rms_eps)
        self.reuse_output = bool(reuse_output)
        self._ws: Dict[int, _Workspace] = {}
        self._ws_shared: Dict[int, _Workspace] = {}
        self.split_widths: Optional[List[int]] = None   # of the layers that run on this one's prologues; None: any

    @classmethod
    def from_prepared(cls, w: "ops.PreparedWeight", ratio: float = 0.05, activation_percentile: float = 100.0,
                      small_m: int = 64, split_k: int = 0, tail_engine: str = "mma", epilogue: str = "none",
                      rms_weight: Optional[torch.Tensor] = None, rms_eps: float = 1e-6,
                      reuse_output: bool = True) -> "SplitLinear":
        """A layer around weights that are already rotated and quantised (e.g. read by `SplitLinear.load`)."""
        if tail_engine not in ("mma", "gather"):
            raise RuntimeError("tail_engine must be 'mma' or 'gather'")
        if epilogue not in ("none", "swiglu"):
            raise RuntimeError("epilogue must be 'none' or 'swiglu'")
        if epilogue == "swiglu" and (tail_engine != "mma" or w.N % 16):
            raise RuntimeError("the SwiGLU epilogue needs the 'mma' tail engine and N % 16 == 0")
        if not w.b_col.is_cuda:
            raise RuntimeError("SplitLinear needs CUDA weights: there is no CPU path")
        R = ops.ceil_ratio_count(int(w.K), float(ratio))
        if R > 0 and tail_engine == "mma" and w.w_rot is None:
            raise RuntimeError("the tensor-core tail needs the rotated bf16 weights (w_rot)")
        if R > 0 and tail_engine == "gather" and w.w_t is None and w.w_rot is not None:
            w.w_t = w.w_rot.t().contiguous()  # the gather engine reads the [K, N] transpose
            w.t_of = (w.w_t, w.w_rot, cls._version(w.w_rot), w.w_rot.data_ptr())
            w.t_made = ops.Made() if w.w_t.device.type == "cuda" else None
        if R > 0 and w.w_t is None and w.w_rot is None:
            raise RuntimeError("a tail needs the rotated bf16 weights (w_rot or w_t)")
        self = cls.__new__(cls)
        self._init(w, ratio, activation_percentile, small_m, split_k, tail_engine, epilogue,
                   None if rms_weight is None else rms_weight.detach().to(device=w.b_col.device, dtype=torch.bfloat16).contiguous(),
                   rms_eps, reuse_output)
        return self

    def save(self, path, policy_entry: Optional[dict] = None) -> None:
        """Writes the prepared weights (packed INT4, scales, rotated bf16 rows, bias) and what the layer fuses around
        them (the epilogue kind, the RMSNorm weight and epsilon) to a `.tqw` file."""
        from . import weights_io
        weights_io.save_prepared(path, self.w, ratio=self.ratio, activation_percentile=self.activation_percentile,
                                 policy_entry=policy_entry, epilogue=self.epilogue, rms_weight=self.rms_weight,
                                 rms_eps=self.rms_eps)

    @classmethod
    def load(cls, path, device="cuda", ratio: Optional[float] = None, tail_engine: str = "mma", small_m: int = 64,
             split_k: int = 0, policy_entry: Optional[dict] = None) -> "SplitLinear":
        """Reads a `.tqw` file; ratio, percentile, epilogue and fused norm default to the ones stored in it."""
        from . import weights_io
        h = weights_io.read_header(path)
        w = weights_io.load_prepared(path, device, need_w_t=False, keep_w_rot=True, expect_policy_entry=policy_entry)
        r = h.get("ratio") if ratio is None else ratio
        return cls.from_prepared(w, ratio=0.0 if r is None else float(r),
                                 activation_percentile=float(h.get("activation_percentile") or 100.0),
                                 small_m=small_m, split_k=split_k, tail_engine=tail_engine,
                                 epilogue=h.get("epilogue") or "none",
                                 rms_weight=weights_io.load_extra(path, "rms_weight", device),
                                 rms_eps=float(h.get("rms_eps") or 1e-6))

    # Estimates in us of the whole linear at few rows, by engine.  The decode kernel reads only the M R tail rows it needs, the
    # fused kernel streams all of the bf16 weights.  Fits to 2880 timings at 1..32 rows of N = 256..28672, K = 512..14336,
    # R = 0.01..0.1 K, half of them with the weights in L2; each grows faster with M than the one after it, so a layer goes
    # from the one kernel over the two to the fused one and never back.  The choice is 0.6 % behind the best on average.
    def _decode_us(self, M: int, apart: bool) -> float:
        """`apart`: the tail sums in a kernel of their own, which reads 512 bytes of a weight row at a time where the decode
        kernel's CTAs read 32 or 64: ahead once the row pieces outweigh a launch and the entries one CTA goes through
        (N = 24576, R = 205: 28 / 29 us at 2 rows, 64 / 36 at 8; N = K = 4096: 14 / 18 at 4, 20 / 18 at 8)."""
        N, K, R, wide = self.N, self.K, self.R, max(1.0, self.N / 4096)
        if apart:
            return 7.14 + 4.79e-4 * K + 9.66e-8 * N * K + 0.0206 * R + (0.14 * M + 6.06e-4 * M * R) * wide
        return 5.87 + 4.72e-4 * K + 5.87e-8 * N * K + (0.342 * M + 0.00374 * M * R) * wide

    def _fused_us(self, M: int) -> float:
        return 5.83e-4 * self.K + max(7.34, 3.46 + 3.73e-7 * self.N * self.K) + 0.0209 * M

    def _tail_apart(self, M: int) -> bool:
        """Whether the decode engine sums the tails in their own kernel (the one kernel takes eight rows with a tail, the
        other one 8192 entries; same bits).  At two rows the third launch costs what it saves: N = 28672, R = 205 30.3 us
        either way in a graph, a layer called launch by launch 2 % slower."""
        if M > 8 or M <= 2 or self.R > 8192:
            return M > 8
        return self._decode_us(M, True) < self._decode_us(M, False)

    def _use_mma(self, M: int) -> bool:
        if self.tail_engine != "mma":
            return False
        if M > min(self.small_m, 32):
            return True
        if not self.R:  # 7.2 / 7.3 us at 16 rows of N = 256, K = 4096; 12.9 / 11.4 at 8, 9.8 / 11.3 at 4 of N = 12288
            return M > (16 if self.N <= 4096 and self.K <= 4096 else 8)
        decode = self._decode_us(M, True)
        return self._fused_us(M) < (decode if M > 8 else min(decode, self._decode_us(M, False)))

    @property
    def N_out(self) -> int:
        return self.N // 2 if self.epilogue == "swiglu" else self.N

    def _engine(self, M: int) -> int:
        if self._use_mma(M):
            return _lib.TQ_LINEAR_FUSED
        return _lib.TQ_LINEAR_DECODE if M <= self.small_m else _lib.TQ_LINEAR_GATHER

    def _provide(self, ws: _Workspace, shared: bool) -> None:
        """Has `ws` show what this layer's forward reads, or with `shared` what any layer on the same prologue may read (a
        layer with the exact-order engine only shares with its like).  The 2:4-sparse form is for layers of any width too, unless
        `split_widths` says which ones follow: then it is there where one of them takes it.  Asked when a forward follows a
        prologue or the other way round, and again under another forced kernel."""
        any_width = shared and self.tail_engine == "mma"
        if any_width and self.split_widths:
            asked = [self._ask(ws, n, False) for n in self.split_widths]
            sparse = any(s for _, s in asked)
            bits, _ = self._ask(ws, self.N, True, sparse)
            for b, _ in asked:
                bits |= b
        else:
            bits, sparse = self._ask(ws, self.N, any_width)
        now = ops.gemm_pair_mode_changes
        if sparse and not shared and not self._follow_w_rot():   # (a captured call without the transpose: the CTA pairs, for now)
            bits, sparse = self._ask(ws, self.N, False, False)
            now = -1
        ws.show(bits, sparse)
        ws.forward_for, ws.shared_for = (-1, now) if shared else (now, -1)

    def _ask(self, ws: _Workspace, N: int, any_width: bool, sparse: Optional[bool] = None) -> Tuple[int, bool]:
        """Prologue outputs for a layer of N channels (`any_width`: for others too), and whether the 2:4-sparse form is one
        (`sparse`: as given)."""
        lib = _lib.load()
        c = _lib.LinearCall(M=ws.M, N=N, K=self.K, R=self.R, had_kind=self.w.had_kind, engine=ws.engine,
                            act=int(self.epilogue == "swiglu"))
        if sparse is None:
            sparse = ws.engine == _lib.TQ_LINEAR_FUSED and lib.tq_linear_sparse(ctypes.byref(c), int(any_width)) > 0
        c.sp_val = 1 if sparse else None   # (asks for what is needed beside it)
        bits = lib.tq_linear_outputs(ctypes.byref(c), int(any_width))
        if bits < 0:
            _lib.check(bits, self._what(ws.M))
        return bits, sparse

    def serves(self, ws: _Workspace, N: int) -> bool:
        """Whether the prologue outputs in `ws` are what a layer of N channels takes, a width not in `split_widths` so far.  If
        not, the next prologue's are."""
        self.split_widths.append(N)
        bits, sparse = self._ask(ws, N, False) if ws.M > 64 else (0, False)
        for w in self._ws.values():
            w.shared_for = -1
        return not (bits & ~ws.outputs or (sparse and ws.pro.sparse is None))

    def _new_workspace(self, M: int, with_pro: bool) -> _Workspace:
        engine = self._engine(M)
        with_tail = self.R > 0 and (engine == _lib.TQ_LINEAR_GATHER or
                                    (engine == _lib.TQ_LINEAR_DECODE and self._tail_apart(M)))
        return _Workspace(M, self.N, self.K, self.R, self.w.b_col.device, engine, self.N_out, with_pro, with_tail)

    def _workspace(self, M: int, shared: bool) -> _Workspace:
        ws = self._ws.get(M)
        if ws is None:
            ws = self._ws[M] = self._new_workspace(M, True)
        if (ws.shared_for if shared else ws.forward_for) != ops.gemm_pair_mode_changes:
            self._provide(ws, shared)
        return ws

    def workspace(self, M: int, shared: bool = True) -> _Workspace:
        """The buffers for `M` rows, with room for every prologue output that a layer on them may read (`shared=False`: with
        those of this layer's forward)."""
        return self._workspace(M, shared)

    def _own_buffers(self, ws: _Workspace, M: int) -> _Workspace:
        """Output and scratch of THIS layer for a prologue workspace that may belong to another layer."""
        if self._ws.get(M) is ws:
            return ws
        if (ws.K, ws.R, ws.M) != (self.K, self.R, M) or (ws.pro.a_q8 if self._use_mma(M) else ws.pro.a_pack) is None:
            raise RuntimeError("a shared prologue needs the same K, R, row count and operand format in both layers")
        own = self._ws_shared.get(M)
        if own is None:
            own = self._ws_shared[M] = self._new_workspace(M, False)
        return own

    def prepare_decode(self) -> None:
        """Builds the [K, N] transpose of the rotated weights that the small-M tail reads, ahead of the first small-M
        forward (which otherwise builds it: an allocation inside that call).  Not inside a stream capture: nothing would have
        written it before the first replay, and every replay would write it again."""
        if self.R:
            self._follow_w_rot()

    def refresh(self) -> None:
        """Makes the [K, N] transpose again, where there is one, after `w_rot` was written by something that its version counter
        does not see: collectives (`torch.distributed.broadcast`, `all_reduce`), `.data.copy_()`, raw pointers, and every
        write to tensors made in inference mode.  In the same memory, so that captured graphs follow; not inside a capture.
        Nothing else of a layer is a copy."""
        w = self.w
        if self.R == 0 or w.w_t is None or w.w_rot is None:
            return
        if self._capturing():
            raise RuntimeError("refresh() cannot run inside a stream capture")
        self._make_transpose(w.w_t)

    @staticmethod
    def _capturing() -> bool:
        return _lib.load().tq_stream_capture_id(ops._stream()) != 0

    def _transposed(self, into: Optional[torch.Tensor] = None) -> torch.Tensor:
        r = self.w.w_rot
        if r.device.type == "cuda" and r.is_contiguous():
            return ops.transpose_bf16(r, into)
        return r.t().contiguous() if into is None else into.copy_(r.t())

    def _make_transpose(self, into: Optional[torch.Tensor] = None) -> None:
        t = self._transposed(into)
        self.w.t_made = ops.Made() if t.device.type == "cuda" else None
        self.w.w_t = t

    @staticmethod
    def _version(t: Optional[torch.Tensor]) -> int:
        return -1 if t is None or t.is_inference() else t._version

    def _rot_version(self) -> int:
        return self._version(self.w.w_rot)

    def _follow_w_rot(self) -> bool:
        """Has `w_t` be there and, from the first call that finds it there, in line with `w_rot`: it is made again when `w_rot` was
        replaced or changed since, in the same memory where `w_rot` is the same tensor (a graph captured before names both).
        One that was replaced with it counts as its transpose.  False where it would have to be made inside a stream capture:
        that call does without, and the next one outside makes it."""
        w, rot = self.w, self.w.w_rot
        if rot is None:
            return w.w_t is not None
        version, address, (t, of, v, place) = self._rot_version(), rot.data_ptr(), w.t_of
        if w.w_t is t and rot is of and version == v and address == place:
            return True
        with _MAKING:   # (threads on streams of their own: one of them makes it, and says so last)
            t, of, v, place = w.t_of
            changed = w.w_t is not None and w.w_t is t and (rot is not of or (version, address) != (v, place))
            if (changed or w.w_t is None) and self._capturing():
                return False
            if changed:
                same = rot is of and tuple(t.shape) == tuple(reversed(rot.shape)) and t.dtype == rot.dtype and t.device == rot.device
                self._make_transpose(t if same else None)
            elif w.w_t is None:
                self._make_transpose()
            w.t_of = (w.w_t, rot, version, address)
        return True

    def _described(self, own: _Workspace) -> bool:
        """Whether `own.call` still names what this layer consists of.  All of it can be replaced between two forwards, and a
        tensor's storage can move under it (`.data = ...`, offloading): objects and addresses are compared on every call,
        half a microsecond where filling the description in again takes ten."""
        w = self.w
        b, c, r, t, i, g, kind, rank, eps, act, pb, pc, pr, pt, pi, pg = own.call_src
        return (b is w.b_col and b.data_ptr() == pb and c is w.w_scale and c.data_ptr() == pc
                and r is w.w_rot and (r is None or r.data_ptr() == pr) and t is w.w_t and (t is None or t.data_ptr() == pt)
                and i is w.bias and (i is None or i.data_ptr() == pi)
                and g is self.rms_weight and (g is None or g.data_ptr() == pg)
                and (own.rot_version is None or own.rot_version == r._version)
                and kind == w.had_kind and rank == self.descending_rank and eps == self.rms_eps and act == self.epilogue)

    def _check_parts(self, engine: int, w_t: Optional[torch.Tensor], reads_t: bool) -> None:
        """Types, layout and sizes of what a forward reads (`w_t`: the transpose it is given): the kernels take it for granted."""
        w, N, K = self.w, self.N, self.K
        ops._check_cuda(w.b_col, "b_col", torch.uint8)
        ops._check(tuple(w.b_col.shape) == (N, K // 2), "b_col must be [N, K/2]")
        ops._check_cuda(w.w_scale, "w_scale", torch.float32)
        ops._check(w.w_scale.numel() >= N, "w_scale must have N elements")
        if self.R and engine == _lib.TQ_LINEAR_FUSED:
            ops._check_cuda(w.w_rot, "w_rot", torch.bfloat16)
            ops._check(tuple(w.w_rot.shape) == (N, K), "w_rot must be [N, K]")
        if reads_t:
            ops._check_cuda(w_t, "w_t", torch.bfloat16)
            ops._check(tuple(w_t.shape) == (K, N), "w_t must be [K, N]")
        if w.bias is not None:
            ops._check_cuda(w.bias, "bias", torch.float32)
            ops._check(w.bias.numel() >= N, "bias must have N elements")
        if self.rms_weight is not None:
            ops._check_cuda(self.rms_weight, "rms_weight", torch.bfloat16)
            ops._check(self.rms_weight.numel() == K, "rms_weight must have K elements")

    def _call(self, own: _Workspace, pro: "ops.PrologueOut"):
        """Reference to the description of this layer's forward: prologue outputs `pro` (own or another layer's), output side
        `own`."""
        if own.call is not None and own.call_pro is pro and self._described(own):
            return own.call
        own.rot_version = own.call = None   # (a part that is refused must not leave the former description in force)
        w, p = self.w, ops._ptr
        keep, w_t = True, w.w_t
        reads_t = self.R > 0 and (own.engine != _lib.TQ_LINEAR_FUSED or (pro.sparse is not None and ops.takes_sparse(
            own.M, self.N, self.K, self.R, w.had_kind, int(self.epilogue == "swiglu"))))
        if reads_t:
            keep, w_t = self._follow_w_rot(), w.w_t
            if not keep:   # in a stream capture: the sparse GEMM reads `w_rot`, the others a transpose for this call of it only
                w_t = self._transposed() if own.engine != _lib.TQ_LINEAR_FUSED and w.w_rot is not None else None
            else:
                if w.w_rot is not None and not w.w_rot.is_inference():
                    own.rot_version = w.t_of[2]
                if w.t_made is not None:
                    w.t_made.order()
        elif pro.sparse is not None and w_t is w.t_of[0]:
            w_t = None   # (where the sparse form is all there is, `w_rot` is what is certain to be in line)
        self._check_parts(own.engine, w_t, reads_t and (keep or own.engine != _lib.TQ_LINEAR_FUSED))
        own.call_pro = pro if keep else None
        own.call_t = w_t   # (lives as long as its address is in `call`)
        src = (w.b_col, w.w_scale, w.w_rot, w.w_t, w.bias, self.rms_weight)
        own.call_src = (*src, w.had_kind, self.descending_rank, self.rms_eps, self.epilogue, *map(p, src))
        own.call = ctypes.byref(_lib.LinearCall(
            M=own.M, N=self.N, K=self.K, R=self.R, had_kind=w.had_kind, descending_rank=self.descending_rank,
            engine=own.engine, act=1 if self.epilogue == "swiglu" else 0,
            tail_ld=pro.tail_idx.shape[1] if pro.tail_idx is not None else 0,
            ptr_ld=pro.tail_ptr.shape[1] if pro.tail_ptr is not None else 0, eps=ops.EPS, rms_eps=self.rms_eps,
            b_col=p(w.b_col), w_scale=p(w.w_scale), w_rot=p(w.w_rot), w_t=p(w_t), bias=p(w.bias),
            rms_weight=p(self.rms_weight), a_pack=p(pro.a_pack), a_q8=p(pro.a_q8), body_scale=p(pro.body_scale),
            top_scale=p(pro.top_scale), tail_idx16=p(pro.tail_idx), tail_val=p(pro.tail_val), tail_ptr=p(pro.tail_ptr),
            tail_rec=p(pro.tail_rec), tail_cnt=p(pro.tail_cnt), tail_dense=p(pro.tail_dense), tail=p(own.tail),
            **({} if pro.sparse is None else dict(zip(ops.SPARSE_FIELDS, map(p, pro.sparse)), sp_over_ld=pro.sparse[3].shape[1]))))
        return own.call

    def _what(self, M: int) -> str:
        return f"SplitLinear(M={M}, N={self.N}, K={self.K}, R={self.R}, had_kind={self.w.had_kind})"

    def prologue(self, x2d: torch.Tensor) -> _Workspace:
        ops._check_cuda(x2d, "x", torch.bfloat16)
        ops._check(x2d.dim() == 2 and x2d.shape[1] == self.K, "x must be [M, K]")
        ws = self.workspace(x2d.shape[0])
        rc = _lib.load().tq_linear_prologue(self._call(ws, ws.pro), x2d.data_ptr(), ops._stream())
        if rc:
            _lib.check(rc, self._what(ws.M))
        return ws

    def compute(self, ws: _Workspace, M: int, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """GEMM + tail for a workspace whose prologue outputs are filled.  `ws` may be ANOTHER layer's workspace
        (shared-prologue use: several linears with the same K, R, rank and rotation run `compute` on one prologue,
        the way the reference shares one prepare between q/k/v and gate/up:
        tools/bench_prefill_bf16_romeoquarotdense_split_total_v61_sharedprepare.py:124-134); the output then goes to
        this layer's own buffer of its own width, or to `out`."""
        own = self._own_buffers(ws, M)
        if out is None:
            out = own.out
        else:
            ops._check_cuda(out, "out", torch.bfloat16)
            ops._check(out.numel() >= M * self.N_out, "out too small")
        rc = _lib.load().tq_linear_compute(self._call(own, ws.pro), out.data_ptr(), ops._stream())
        if rc:
            _lib.check(rc, self._what(M))
        return out

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        shape = x.shape
        if x.dtype is not torch.bfloat16:
            x = x.to(torch.bfloat16)
        if shape[-1] != self.K or not x.is_contiguous():
            x = x.reshape(-1, self.K).contiguous()
        if not x.is_cuda:
            raise RuntimeError("x must be a CUDA tensor")
        M = x.numel() // self.K
        ws = self._ws.get(M)
        if ws is None or ws.forward_for != ops.gemm_pair_mode_changes:
            ws = self._workspace(M, False)
        call = ws.call
        if call is None or ws.call_pro is not ws.pro or not self._described(ws):
            call = self._call(ws, ws.pro)
        y = ws.out if self.reuse_output else torch.empty_like(ws.out)
        rc = _lib.load().tq_linear_forward(call, x.data_ptr(), y.data_ptr(), ops._stream())
        if rc:
            _lib.check(rc, self._what(M))
        return y.view(*shape[:-1], self.N_out)

    __call__ = forward


# ------------------------------------------------------------------------------------------ adapter callable
class _Entry:
    __slots__ = ("lin", "wref", "bref", "shape", "ratio")


_CACHE: "OrderedDict[Tuple, _Entry]" = OrderedDict()
_CACHE_MAX = 1024        # prepared layers kept (a 36-layer model has 252 target linears)
_SHARED: Dict[Tuple, Tuple] = {}  # (input, shape of the split, stream, capture) -> (x weakref, workspace, its layer)


def _drop(key) -> None:
    _CACHE.pop(key, None)


def clear_cache() -> None:
    """Forgets every layer prepared by `split_linear_forward` (and frees their device memory)."""
    _CACHE.clear()
    _SHARED.clear()


def _cached_layer(weight: torch.Tensor, bias: Optional[torch.Tensor], ratio: float) -> SplitLinear:
    key = (weight.device.index, weight.data_ptr(), weight._version, tuple(weight.shape), float(ratio),
           None if bias is None else (bias.data_ptr(), bias._version))
    e = _CACHE.get(key)
    # an address can be handed out again by the caching allocator after its tensor died: the entry only counts
    # if it was built from THIS tensor object
    if e is not None and e.wref() is weight and (bias is None or (e.bref is not None and e.bref() is bias)):
        _CACHE.move_to_end(key)
        return e.lin
    e = _Entry()
    e.lin = SplitLinear(weight, bias, ratio, reuse_output=True)
    e.lin.split_widths = [e.lin.N]   # (others are added as they come)
    e.wref = weakref.ref(weight, lambda _r, k=key: _drop(k))  # the entry goes when the weight does
    e.bref = None if bias is None else weakref.ref(bias)
    _CACHE[key] = e
    _CACHE.move_to_end(key)
    while len(_CACHE) > _CACHE_MAX:
        _CACHE.popitem(last=False)
    return e.lin


def split_linear_forward(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                         ratio: float = 0.05, split_ratio: Optional[float] = None) -> torch.Tensor:
    """Callable the reference's adapter binds (tools/split_backend_adapter_v1.py:92-116): called as
    fn(x [M,K], weight [N,K], bias=, ratio=) on every forward with the RAW weight, so prepared weights are cached
    per weight tensor (object identity, version, shape, ratio; an entry dies with its weight, the cache is
    bounded).  Returns a NEW [M, N] tensor in x's dtype, like the nn.Linear it stands in for.

    Consecutive calls on the SAME input tensor by layers with the same K, R and rotation -- q/k/v, gate/up of a
    model patched module by module -- share one prologue, the reference's shared prepare
    (tools/bench_prefill_bf16_romeoquarotdense_split_total_v61_sharedprepare.py:221-261)."""
    if split_ratio is not None:
        ratio = split_ratio
    if bias is not None and not torch.is_tensor(bias):  # the adapter's positional form fn(x, W, ratio)
        ratio, bias = float(bias), None
    if weight.dim() != 2 or x.shape[-1] != weight.shape[1]:
        raise RuntimeError(f"weight must be [N, K] with K = x.shape[-1]; got {tuple(weight.shape)} for x {tuple(x.shape)}")
    lin = _cached_layer(weight, bias, ratio)
    x2d = x.reshape(-1, lin.K)
    if x2d.dtype != torch.bfloat16:
        x2d = x2d.to(torch.bfloat16)
    x2d = x2d.contiguous()
    M = x2d.shape[0]
    stream = ops._stream()
    # Only an input that is used as it is can be recognised again, and only one whose in-place changes are counted (those
    # made in inference mode are not).
    known = x2d.data_ptr() == x.data_ptr() and not x.is_inference()
    # (a graph has to contain the prologue of its linears: one that ran before the capture, or in another, is none of it)
    skey = (x.device.index, x2d.data_ptr(), x._version if known else 0, M, lin.K, lin.R, lin.descending_rank, lin.w.had_kind, stream,
            _lib.load().tq_stream_capture_id(stream))
    hit = _SHARED.get(skey) if known else None
    owner = hit[2]() if hit is not None and hit[0]() is x else None
    if owner is not None:
        ws = hit[1]
        known_widths = owner.split_widths
        if known_widths is not None and lin.N not in known_widths and not owner.serves(ws, lin.N):   # (a width's first time)
            ws = owner.prologue(x2d)
    else:
        _SHARED.clear()   # one entry: the prologue outputs live in a workspace that the next prologue of that layer
        ws = lin.prologue(x2d)                    # overwrites, whatever its input
        if known:
            _SHARED[skey] = (weakref.ref(x), ws, weakref.ref(lin))
    y = lin.compute(ws, M, torch.empty((M, lin.N_out), dtype=torch.bfloat16, device=x2d.device))
    y = y.view(*x.shape[:-1], lin.N_out)
    return y if y.dtype == x.dtype else y.to(x.dtype)
