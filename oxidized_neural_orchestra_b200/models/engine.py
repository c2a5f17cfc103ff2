"""GPU training engine: explicit forward/backward over flat f32 parameters in HBM.

The engine is the B200 counterpart of the reference's ``Sequential`` + ``ParamManager``
(machine_learning/src/arch/sequential.rs:43-148, machine_learning/src/param_manager.rs:61-198):

* parameters and gradients are two flat f32 vectors in the reference's external layout
  (per layer ``W[in,out]`` row-major then ``b[out]``; conv ``K[F][C][k][k]`` then ``b[F]``), so that
  collectives, optimizers and the safetensors export all work on the same buffer;
* layers are views (offset tables) into those vectors;
* every GEMM runs on the tcgen05 kernel; operands the tensor cores cannot address directly from the
  flat vector (unaligned rows, bf16 tiles) are "compute copies" that
  ``refresh()`` regenerates after each parameter update;
* there is no autograd: each layer contributes explicit forward, dgrad and wgrad launches, and a
  whole mini-batch step is a fixed kernel sequence that can be captured in a CUDA graph.

Tile dtype ``tf32`` keeps every tensor in f32, ``bf16`` keeps bf16 activations and deltas. Operands whose
reduction does not run along their rows are read as MN-major tiles, so no transposed copies exist.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass, field

import torch

from ..ops import _lib
from ..ops import elementwise as ew
from ..ops.gemm import ACT, _workspace, gemm


def _up(n: int, m: int = 16) -> int:
    return (n + m - 1) // m * m


@dataclass
class LayerPlan:
    kind: str                       # dense | conv | pool
    in_features: int
    out_features: int
    act: str | None = None
    act_param: float = 0.0
    w_off: int = 0                  # offset of W in the flat vector
    b_off: int = 0                  # offset of b
    n_params: int = 0
    extra: dict = field(default_factory=dict)


def layer_param_count(spec: dict) -> int:
    if spec["kind"] == "dense":
        return (spec["in"] + 1) * spec["out"]
    if spec["kind"] == "conv":
        f, c, k = spec["kernel_dim"]
        return f * c * k * k + f
    return 0


def on_device_rows(t: torch.Tensor, rows: int, width: int) -> bool:
    """Whether kernels may read the first ``rows`` rows where they are."""
    return t.is_cuda and t.dtype == torch.float32 and t.dim() == 2 and t.shape[0] >= rows and t.shape[1] == width and t.stride(1) == 1


class Beside:
    """Launches on a second stream beside the ones that follow on ``main``: ``mark()`` where their inputs exist, ``on()`` for the
    stream to launch on, ``join()`` where their results are needed. Without a second stream everything stays on ``main``."""

    def __init__(self, main, side):
        self.main = main if main is not None else torch.cuda.current_stream()
        self.side, self.used, self.ev = side, False, None

    def mark(self, wanted: bool) -> None:
        self.ev = None
        if self.side is not None and wanted:
            self.ev = torch.cuda.Event()
            self.ev.record(self.main)

    def on(self):
        if self.ev is None:
            return self.main
        self.side.wait_event(self.ev)
        self.used = True
        return self.side

    def join(self) -> None:
        if self.used:
            self.main.wait_stream(self.side)
            self.used = False


class GpuEngine:
    """Forward/backward of a dense network for one fixed maximum batch size on one GPU."""

    def __init__(self, layers: list[dict], *, batch_size: int, tile_dtype: str, loss: str,
                 params: torch.Tensor, grads: torch.Tensor, params_bf16: torch.Tensor | None = None,
                 leaky_relu_exact: bool = True, device=None, bias_from_shadow: bool = False,
                 input_grad: bool = False, final: bool = True):
        self.bias_from_shadow = bias_from_shadow
        # final = False: a dense block in the middle of a network (convolutions follow). Its last layer then writes its
        # activation into ``out_act`` like any inner layer, and backward starts from ``d[-1]``, which whoever consumes
        # ``out_act`` fills with the gradient w.r.t. that layer's pre-activation.
        self.final = final
        self.input_grad = input_grad  # also produce d[0], the gradient w.r.t. the input batch
        # One order of additions for every sum of a step, from version to version (GEMMs here; bias sums and a one-channel first
        # layer's weight gradient have it for all bf16 matrices). Kept by networks with bf16 tiles that have ReLUs or convolutions:
        # their activations and deltas are rounded to 8 bits after every layer, a ReLU whose pre-activation lies within that of zero
        # flips, and a gradient that few samples make up then moves by percents. Another order of the same f32 sums moved single
        # entries of the moments by 1.05 of their size within two steps of a 28 x 28 network (32, 64, 64 filters, 2048 images), and by
        # 2.2 in a deep ReLU network at batch 27. Smooth activations do not amplify so (0.3 at most over 120 drawn networks), nor
        # do tf32 tiles, which round to 10 bits and only as operands: these take whatever form is the fastest.
        self.fixed_order = tile_dtype == "bf16" and any(l.get("act") and l["act"][0] == "relu" for l in layers)
        self.max_ctas = 0             # CTAs a GEMM of this engine may use (0 = one per SM); lowered while other kernels need SMs
        self.push = None              # weight-gradient tiles added into the owners' f32 accumulators (see backward)
        self.wire16 = None            # weight-gradient tiles stored as 16-bit values into the owners' slabs
        # A weight gradient waits for nothing but its layer's delta: with a second stream (``side``, the caller's to give) it runs
        # beside the input gradients of the layers below. Of a small layer either fills a few SMs, of a large one the last wave and
        # the epilogue of one leave room for the other: 26 random networks 1.00 to 1.29 times faster, from 0.01 M to 17 G
        # multiply-adds a layer (lenet5 step 150.8 -> 126.6 us, ragged 98 -> 89, 992 x 2448 wide 767 -> 652).
        self.side = None
        self.report_to = None         # pinned float64[1] the batch's loss goes to
        self.apply_plan = None        # optimizer applied by the weight-gradient GEMM's epilogue, per layer
        self.gates = None             # per layer: flags its forward GEMM waits on before it loads the layer's weights
        if tile_dtype not in ("tf32", "bf16"):
            raise ValueError("tile_dtype must be 'tf32' or 'bf16'")
        self.dev = device or params.device
        if self.dev.type != "cuda":
            raise RuntimeError("GpuEngine needs a CUDA device; CPU runs use the C++ oracle engine")
        self.bf16 = tile_dtype == "bf16"
        self.B = batch_size
        self.loss = loss
        self.relu_quirk = not leaky_relu_exact
        self.params, self.grads, self.params_bf16 = params, grads, params_bf16
        self.plans: list[LayerPlan] = []
        off = 0
        for sp in layers:
            if sp["kind"] != "dense":
                raise NotImplementedError("GpuEngine handles dense layers; see ConvEngine for conv/pool")
            act = sp.get("act")
            pl = LayerPlan("dense", sp["in"], sp["out"], act[0] if act else None, act[1] if act else 0.0)
            pl.w_off, pl.b_off = off, off + sp["in"] * sp["out"]
            pl.n_params = (sp["in"] + 1) * sp["out"]
            off += pl.n_params
            self.plans.append(pl)
        self.n_params = off
        if params.numel() < off or grads.numel() < off:
            raise ValueError("flat parameter/gradient buffers are too small")
        # softmax on the last layer is fused into the loss kernel; on any other layer it is a row-wise pass of its own
        # after the GEMM (forward) and before the next GEMM's operand is formed (Jacobian-vector product in backward)
        self.softmax_last = self.final and self.plans[-1].act == "softmax"
        if not self.final and self.plans[-1].act in ("softmax", "gelu"):
            raise NotImplementedError("a dense layer followed by a convolution needs a relu / sigmoid / tanh / linear activation")
        self._alloc()
        # The layers from here on run as two launches (0: the whole network; None: none do). See _small_fits.
        self.small = self._small_fits()
        self._stale = False                   # the operand copies of those layers' weights have not been made (they need none)

    # ------------------------------------------------------------------------------------------
    def _alloc(self) -> None:
        dev, B = self.dev, self.B
        cd = torch.bfloat16 if self.bf16 else torch.float32
        f32 = torch.float32
        z = lambda r, c, dt: torch.zeros(r, c, device=dev, dtype=dt)
        L = self.plans
        feats = [L[0].in_features] + [p.out_features for p in L]
        self.lds = [_up(f) for f in feats]
        # activations a[0] = input batch, a[l+1] = output of layer l
        self.a = [z(B, self.lds[i], cd) for i in range(len(feats) - 1)]
        self.logits = z(B, self.lds[-1], f32)
        self.d = [z(B, self.lds[0], cd) if self.input_grad else None] + [z(B, self.lds[i], cd) for i in range(1, len(feats))]
        self.zpre = [None] * len(feats)
        self.soft_tmp = [None] * len(feats)       # f32 scratch of an inner softmax layer: pre-activations, then d/d(output)
        for l, pl in enumerate(L):
            if pl.act == "gelu":
                self.zpre[l + 1] = z(B, self.lds[l + 1], cd)
            if pl.act == "softmax" and l < len(L) - 1:
                self.soft_tmp[l + 1] = z(B, self.lds[l + 1], f32)
        # MN-major operands let every GEMM read activations, deltas and weights as they are stored, in either tile type. (tf32
        # once took K-major tiles from transposed copies of all three: a weight-gradient product is faster that way, 58.7 against
        # 66.7 us at 4096 x 4096 x 1024, but writing the copies cost more everywhere: wide MLP step 763 against 705 us, 24 random
        # networks 1.00 to 1.19 times slower.)
        self.out_act = None if self.final else z(B, self.lds[-1], cd)
        self.ybuf = z(B, _up(feats[-1]), f32)
        self.loss_sum = torch.zeros(1, device=dev, dtype=torch.float64)
        self.correct = torch.zeros(1, device=dev, dtype=torch.int32)
        self.status = torch.zeros(1, device=dev, dtype=torch.int32)
        self.small_scratch = torch.zeros(_lib.DENSE_SCRATCH, device=dev, dtype=torch.uint8)
        # weight operands
        self.w_k, self.w_copy_needed = [], []
        for pl in L:
            i, o = pl.in_features, pl.out_features
            esz_mult = 8 if self.bf16 else 4
            flat = self.params_bf16 if self.bf16 else self.params
            direct = flat is not None and o % esz_mult == 0 and pl.w_off % esz_mult == 0 and \
                (flat.data_ptr() + pl.w_off * flat.element_size()) % 16 == 0
            if direct:
                self.w_k.append(flat[pl.w_off:pl.w_off + i * o].view(i, o))
                self.w_copy_needed.append(False)
            else:
                self.w_k.append(z(i, _up(o), cd)[:, :o])
                self.w_copy_needed.append(True)

    def set_side(self, stream) -> None:
        """A second stream for launches beside those of the step. It gets its split-K workspace here: without one its products would
        take the library's only static buffer, which those of the other stream may be using."""
        if stream is not None and _workspace(self.dev, stream) is None:
            raise RuntimeError("set_side during a stream capture: the second stream's workspace cannot be allocated")
        self.side = stream

    def set_report(self, host: torch.Tensor | None) -> None:
        """``step`` leaves the batch's loss in ``host`` (pinned float64[1])."""
        self.report_to = host

    def _gemm(self, *args, **kw) -> None:
        gemm(*args, max_ctas=self.max_ctas, fixed_order=self.fixed_order, **kw)

    def w_view(self, l: int) -> torch.Tensor:
        pl = self.plans[l]
        return self.params[pl.w_off:pl.w_off + pl.in_features * pl.out_features].view(pl.in_features, pl.out_features)

    @property
    def needs_f32_params(self) -> bool:
        """False when every operand the engine reads comes from the bf16 shadow (weights used in place
        and biases read as bf16): then only the owner of a range needs its f32 master."""
        return not (self.bf16 and self.bias_from_shadow and self.params_bf16 is not None
                    and not any(self.w_copy_needed))

    def b_view(self, l: int) -> torch.Tensor:
        pl = self.plans[l]
        if not self.needs_f32_params:
            return self.params_bf16[pl.b_off:pl.b_off + pl.out_features]
        return self.params[pl.b_off:pl.b_off + pl.out_features]

    def gw_view(self, l: int) -> torch.Tensor:
        pl = self.plans[l]
        return self.grads[pl.w_off:pl.w_off + pl.in_features * pl.out_features].view(pl.in_features, pl.out_features)

    def gb_view(self, l: int) -> torch.Tensor:
        pl = self.plans[l]
        return self.grads[pl.b_off:pl.b_off + pl.out_features]

    # ------------------------------------------------------------------------------------------
    def refresh(self, stream=None) -> int:
        """Regenerate the compute copies of the weights from the f32 master. Returns #launches."""
        t = self.small_from()
        self._stale = t is not None
        return self._copies(stream, range(len(self.plans) if t is None else t))

    def _copies(self, stream, layers) -> int:
        jobs = [dict(src=self.w_view(l), **{"dst_bf16" if self.bf16 else "dst": self.w_k[l]})
                for l in layers if self.w_copy_needed[l]]
        return ew.rows_jobs(jobs, stream=stream)

    def batch_job(self, x: torch.Tensor, nrows: int, idx: torch.Tensor | None = None) -> dict:
        """``x[idx]`` (f32, [rows, in]) as the first GEMM's A operand: arguments for ``ew.rows``."""
        return dict(src=x, idx=idx, n_rows=nrows, **{"dst_bf16" if self.bf16 else "dst": self.a[0]})

    def load_batch(self, x: torch.Tensor, y: torch.Tensor, nrows: int, idx: torch.Tensor | None = None,
                   stream=None, zero_loss: bool = False) -> int:
        """Stage ``x[idx]`` (f32, [rows, in]) as the first GEMM's A operand and ``y[idx]`` as the labels."""
        jobs = [self.batch_job(x, nrows, idx), dict(src=y, idx=idx, n_rows=nrows, dst=self.ybuf)]
        return ew.rows_jobs(jobs, zero=self.loss_sum if zero_loss else None, stream=stream)

    def forward(self, nrows: int, stream=None, upto: int | None = None) -> int:
        """The layers in front of ``upto`` (None: all)."""
        L, n = self.plans, 0
        if self._stale and upto is None:
            n += self._copies(stream, range(self.small, len(L)))
        for l, pl in enumerate(L[:upto]):
            last = l == len(L) - 1 and self.final
            a_in = self.a[l][:nrows, :pl.in_features]
            inner_softmax = pl.act == "softmax" and not last
            act = None if (pl.act == "softmax") else pl.act
            kw = dict(bias=self.b_view(l), act=act, act_param=pl.act_param, status=self.status, stream=stream)
            if self.gates is not None and self.gates.get(l) is not None:
                kw["gate"] = self.gates[l]      # the layer's weights may still be arriving from their owners
                kw["timeout_ns"] = 10_000_000_000   # the same patience as the fused kernel's barriers: a rank may start late
            if inner_softmax:
                o = pl.out_features
                kw["out"] = self.soft_tmp[l + 1][:nrows, :o]
                self._gemm(a_in, self.w_k[l], b_mn_major=True, **kw)
                ew.softmax_layer(self.soft_tmp[l + 1][:nrows, :o], out=self.a[l + 1][:nrows, :o], stream=stream)
                n += 2
                continue
            if last:
                kw["out"] = self.logits[:nrows, :pl.out_features]
            elif l == len(L) - 1:      # a block in the middle of a network: the activation goes to whoever follows
                kw["out_bf16" if self.bf16 else "out"] = self.out_act[:nrows, :pl.out_features]
            else:
                kw["out_bf16" if self.bf16 else "out"] = self.a[l + 1][:nrows, :pl.out_features]
                if self.zpre[l + 1] is not None:
                    kw["pre"] = self.zpre[l + 1][:nrows, :pl.out_features]
            self._gemm(a_in, self.w_k[l], b_mn_major=True, **kw)
            n += 1
        return n

    def loss_backward(self, nrows: int, stream=None) -> int:
        y = self.ybuf
        pl = self.plans[-1]
        C = pl.out_features
        lg = self.logits[:nrows, :C]
        kw = dict(kind=self.loss, softmax=self.softmax_last, loss_sum=self.loss_sum, correct=self.correct,
                  stream=stream)
        if not self.softmax_last and pl.act is not None:
            kw.update(dact=pl.act, dact_param=pl.act_param, relu_quirk=self.relu_quirk)
        if self.bf16:
            kw["d_bf16"] = self.d[-1][:nrows, :C]
        else:
            kw["d"] = self.d[-1][:nrows, :C]
        ew.loss_backward(lg, y[:nrows, :C], **kw)
        return 1

    def backward(self, nrows: int, accumulate: bool = False, stream=None, after_layer=None, bias_jobs: list | None = None, tail=None) -> int:
        """dgrad + wgrad + bias-grad for every layer; gradients land in the flat gradient vector. ``tail``: the layers from
        ``small`` on have been through ``small_rows``, which returned it; what is left of them are their weight gradients.

        Bias gradients nobody waits for layer by layer are summed in one launch, beside the last weight gradient (or appended to
        ``bias_jobs``, for a caller that has more of them).

        Per layer the input gradient is computed first, so that nothing reads the layer's weights once
        its own gradient is complete: ``after_layer(l)`` may then start synchronising (and overwriting)
        that layer's parameters while the layers below are still running."""
        L, n = self.plans, 0
        beta = 1.0 if accumulate else 0.0
        late: list = [] if bias_jobs is None else bias_jobs

        def bias_grad(l, d, b):
            if after_layer is None:
                late.append((d, self.gb_view(l), b))
                if l > 0 or bias_jobs is not None:
                    return 0
                # every delta exists: all bias gradients at once, beside the last weight gradient. Where that one runs on the second
                # stream itself, beside the input gradient (its mark stays), they follow the input gradient: ahead of it there, 512
                # bf16 samples through two units of convolutions took 139.2 us a step, so 131.3
                if sums is par and par.ev is not None:
                    return ew.colsum_jobs(late, stream=stream)
                sums.mark(True)
                k = ew.colsum_jobs(late, stream=sums.on())
                sums.mark(False)
                return k
            ew.colsum(d, self.gb_view(l), beta=b, stream=stream)
            return 1

        push, wire, app = self.push, self.wire16, self.apply_plan
        if (push is not None or wire is not None or app is not None) and accumulate:
            raise RuntimeError("pushed / fused weight gradients cannot accumulate over several batches")
        # (an owner's or a fused optimizer's weight gradient changes what the input gradient reads: those stay in order)
        par = Beside(stream, self.side if after_layer is None and push is None and wire is None and app is None else None)
        sums = par if par.side is not None else Beside(stream, self.side)
        top = len(L) - 1 if tail is None else self.small - 1
        for l in range(top, -1, -1):
            pl = L[l]
            i, o = pl.in_features, pl.out_features
            d_out = self.d[l + 1][:nrows, :o]
            par.mark(l > 0 or self.input_grad)      # (below the first layer nothing is left to run beside)
            if l == top and tail is not None:
                sums.mark(True)
                self.small_grads(tail, accumulate, sums.on())
                n += 1
                if sums is par:
                    par.mark(l > 0 or self.input_grad)
            elif l == top and self.report_to is not None:
                if sums is not par:
                    sums.mark(True)
                ew.report(self.loss_sum, self.report_to, stream=sums.on())
                n += 1
            if l > 0 or self.input_grad:
                # dgrad through the previous layer's activation: d_{l} = (d_{l+1} W^T) * act'(a_l);
                # for l = 0 this is the raw gradient w.r.t. the input batch (whoever produced the
                # batch applies its own activation derivative)
                prev = L[l - 1] if l > 0 else LayerPlan("input", 0, i)
                stored = self.zpre[l] if prev.act == "gelu" else self.a[l]
                kw = dict(status=self.status, stream=stream)
                if prev.act == "softmax":
                    # the GEMM leaves d/d(softmax output) in f32; the Jacobian-vector product needs whole rows
                    tmp = self.soft_tmp[l][:nrows, :i]
                    self._gemm(d_out, self.w_k[l], out=tmp, **kw)
                    ew.softmax_layer(tmp, p=self.a[l][:nrows, :i], out=self.d[l][:nrows, :i], stream=stream)
                    n += 2
                elif prev.act is not None:
                    kw.update(aux=stored[:nrows, :i], dact=prev.act, dact_param=prev.act_param,
                              relu_quirk=self.relu_quirk)
                if prev.act != "softmax":
                    self._gemm(d_out, self.w_k[l], **{"out_bf16" if self.bf16 else "out": self.d[l][:nrows, :i]}, **kw)
                    n += 1

            def wgrad(r0, r1, **out_kw):     # rows [r0, r1) of dW = A_l^T d
                self._gemm(self.a[l][:nrows, r0:r1], d_out, a_mn_major=True, b_mn_major=True, status=self.status, stream=par.on(),
                           **out_kw)

            if wire is not None:
                # 16-bit gradient wire. "staged": dW leaves the epilogue as bf16 / f16 into this rank's own 16-bit
                # gradient vector (TMA stores to local memory); the caller's after_layer hook then ships the ranges other
                # ranks own with copy-engine transfers while backward goes on. "direct": the epilogue's TMA stores go
                # straight into the slab the owner of those rows keeps for this rank (its window over NVLink).
                k16 = "out_f16" if wire["f16"] else "out_bf16"
                pieces = wire["w"][l]
                if pieces is not None:
                    # into a peer's window the persistent kernel's TMA stores rather than a cluster's plain stores (of a few tiles with
                    # a long reduction the finishing pass of the split still writes plain ones)
                    form = {"cluster": -1} if wire.get("direct") else {}
                    for r0, r1, dst in pieces:
                        wgrad(r0, r1, **{k16: dst}, **form)
                        n += 1
                else:
                    wgrad(0, i, out=self.gw_view(l), any_ld=True)
                    n += 1
                ew.colsum(d_out, self.gb_view(l), beta=0.0, stream=stream)
                n += 1
                for src, dst in wire["cast"][l]:
                    ew.cast16(src, dst, f16=wire["f16"], stream=stream)
                    n += 1
                if after_layer is not None:
                    n += after_layer(l) or 0
                continue
            if app is not None and app.get(l) is not None:
                # this rank owns the whole layer: the epilogue applies the optimizer to the tile it has just
                # computed (master, state, bf16 shadow); the weight gradient itself is never stored
                n += 1 + bias_grad(l, d_out, 0.0)
                wgrad(0, i, apply=app[l])
                if after_layer is not None:
                    n += after_layer(l) or 0
                continue
            if push is not None:
                # weight gradient tiles are added straight into the accumulator of the rank that owns those rows (its
                # window, over NVLink): the reduce-scatter happens inside the GEMM epilogue, tile by tile
                for r0, r1, dst in push["w"][l]:
                    wgrad(r0, r1, out=dst, reduce_out=True)
                    n += 1
                ew.colsum(d_out, self.gb_view(l), beta=0.0, stream=stream)
                ew.push_add(self.gb_view(l), push["b"][l], stream=stream)
                n += 2
                if after_layer is not None:
                    n += after_layer(l) or 0
                continue
            # wgrad: dW[in,out] = A_{l}^T d
            n += 1 + bias_grad(l, d_out, beta)
            wgrad(0, i, out=self.gw_view(l), beta=beta, any_ld=True)
            if after_layer is not None:
                n += after_layer(l) or 0
        sums.join()
        if par is not sums:
            par.join()
        return n

    # ------------------------------------------------------------------------------------------
    def _small_fits(self) -> int | None:
        """The first layer from which on this network's steps run as ``csrc/kernels/dense_step.cu`` has them: tf32 tiles, at most 32
        outputs and 1024 samples, and an eighth of those layers' weights (a quarter above 384 samples) with the activations of 16 or 32
        samples in one SM's shared memory. Two launches against one per layer and product, us a step without the optimizer: of 340 drawn networks
        none is slower that way but two of one layer (74-16 at 967 samples 23.0 against 19.6); 784-128-10 at 32 samples 18.2 against 32.5, 196-94-10 at 167 20.9 / 34.5,
        17-169-74-32 at 578 36.1 / 50.6, 66-263-10 at 682 32.9 / 36.9. The end of a network that does not fit takes the form behind a layer of
        at most 256 and up to 384 samples (behind 68 of 762-68-269-10 at 28 38.5 / 48.7, behind 192 of 225-696-192-10 at 32 42.6 / 46.7;
        behind 606 of 550-606-10 at 13 36.9 / 36.2, behind 318 of 171-152-318-494-10 at 518 85.8 / 78.4)."""
        L = self.plans
        if self.bf16 or not self.final or L[-1].act == "gelu":
            return None
        for t in range(max(0, len(L) - _lib.DENSE_MAX), len(L)):
            if any(p.act == "softmax" for p in L[max(0, t - 1):-1]) or t and (L[t].in_features > 256 or self.B > 384):
                continue
            s = _lib.OnoDenseStep()
            s.rows, s.n_layers = self.B, len(L) - t
            for q, p in zip(s.layer, L[t:]):
                q.n_in, q.n_out, q.act = p.in_features, p.out_features, ACT[None if p.act == "softmax" else p.act]
            s.dx = 1 if t or self.input_grad else None       # (asked about, not written to)
            if _lib.load().ono_dense_step_fits(C.byref(s)):
                return t
        return None

    def small_from(self) -> int | None:
        """``small``, unless something else has to happen to single layers' weights or gradients."""
        return self.small if self.push is None and self.wire16 is None and self.apply_plan is None and self.gates is None else None

    def _small_args(self, x: torch.Tensor, y: torch.Tensor, nrows: int, zero_loss: bool) -> "_lib.OnoDenseStep":
        """``x``: what the first of these layers reads, ``y``: labels; rows on the device, f32, unit inner stride."""
        t = self.small
        s, L, f = _lib.OnoDenseStep(), self.plans[t:], self.params.data_ptr()
        g = self.grads.data_ptr()
        s.x, s.ldx, s.rows, s.n_layers, s.relu_quirk = x.data_ptr(), x.stride(0), nrows, len(L), int(self.relu_quirk)
        for k, p in enumerate(L):
            q, l = s.layer[k], t + k
            q.w, q.b, q.gw, q.gb = f + 4 * p.w_off, f + 4 * p.b_off, g + 4 * p.w_off, g + 4 * p.b_off
            q.n_in, q.n_out = p.in_features, p.out_features
            q.act, q.act_param = ACT[None if p.act == "softmax" else p.act], p.act_param
            if k < len(L) - 1:
                q.a, q.ld_a, q.d, q.ld_d = self.a[l + 1].data_ptr(), self.a[l + 1].stride(0), self.d[l + 1].data_ptr(), self.d[l + 1].stride(0)
        last, o = L[-1], s.loss
        ew.fill_loss(o, nrows, last.out_features, y, self.loss, self.softmax_last, self.loss_sum, self.correct)
        o.d_f32, o.ld_d = self.d[-1].data_ptr(), self.d[-1].stride(0)
        if not self.softmax_last and last.act is not None:
            o.dact, o.dact_param, o.relu_quirk = ACT[last.act], last.act_param, int(self.relu_quirk)
        if t or self.input_grad:
            s.dx, s.ld_dx = self.d[t].data_ptr(), self.d[t].stride(0)
        if t:
            below = self.plans[t - 1]
            aux = self.zpre[t] if below.act == "gelu" else self.a[t]
            s.dx_aux, s.ld_dx_aux, s.dx_act, s.dx_param = aux.data_ptr(), aux.stride(0), ACT[below.act], below.act_param
        s.zero_loss = int(zero_loss)
        s.host_loss = None if self.report_to is None else self.report_to.data_ptr()
        s.scratch = self.small_scratch.data_ptr()
        return s

    def small_rows(self, x, y, nrows: int, stream=None, zero_loss: bool = False):
        """Forward, loss and input gradients in one launch; returns what ``small_grads`` takes."""
        s = self._small_args(x, y, nrows, zero_loss)
        _lib.check(_lib.load().ono_dense_step(C.byref(s), _lib.stream_ptr(stream)), "ono_dense_step")
        return s

    @staticmethod
    def small_grads(s, accumulate: bool, stream=None) -> None:
        """Every weight and bias gradient of the same step in one launch."""
        _lib.check(_lib.load().ono_dense_grads(C.byref(s), 1.0 if accumulate else 0.0, _lib.stream_ptr(stream)), "ono_dense_grads")

    def step(self, x: torch.Tensor, y: torch.Tensor, nrows: int, idx=None, accumulate=False, stream=None,
             after_layer=None, zero_loss: bool = False) -> int:
        """load -> forward -> loss -> backward. Returns the number of kernels launched. The batch's loss is added to
        ``loss_sum`` (which ``zero_loss`` clears first)."""
        t = self.small_from() if after_layer is None else None
        if t is not None:
            x_here = t == 0 and idx is None and on_device_rows(x, nrows, self.plans[0].in_features)
            y_here = idx is None and on_device_rows(y, nrows, self.plans[-1].out_features)
            jobs = ([] if x_here else [self.batch_job(x, nrows, idx)]) + ([] if y_here else [dict(src=y, idx=idx, n_rows=nrows, dst=self.ybuf)])
            n = ew.rows_jobs(jobs, stream=stream) + self.forward(nrows, stream, upto=t) + 1
            s = self.small_rows(x if x_here else self.a[t], y if y_here else self.ybuf, nrows, stream, zero_loss)
            if t == 0:
                self.small_grads(s, accumulate, stream)
                return n + 1
            return n + self.backward(nrows, accumulate, stream, tail=s)
        n = self.load_batch(x, y, nrows, idx, stream, zero_loss)
        n += self.forward(nrows, stream)
        n += self.loss_backward(nrows, stream)
        n += self.backward(nrows, accumulate, stream, after_layer)
        return n
