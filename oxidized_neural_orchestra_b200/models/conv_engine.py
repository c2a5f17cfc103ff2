"""Convolution / pooling layers ahead of the dense stack on the GPU.

The reference runs ``Conv2d`` as per-sample im2col + GEMM and ``MaxPooling`` as a scalar window scan
(machine_learning/src/arch/layers/conv/conv2d.rs:61-190, arch/layers/max_pooling.rs:47-157). Here a
convolution is one batched tcgen05 GEMM ``cols[B*oh*ow, C*k*k] @ K[F, C*k*k]^T`` with bias and activation
in its epilogue, the weight gradient a split-K GEMM over all output pixels of the batch, the input
gradient a GEMM followed by a gather-form col2im. Columns are ordered (ky, kx, c) - channels fastest - so
that the gathers read and write contiguous runs; the kernel tensor ``K[F][C][k][k]`` is permuted into that
order at every parameter refresh and the weight gradient is permuted back into the flat gradient vector. Image activations are pixel-major ``[B*H*W, ld]``; the flattened
NCHW order dense layers expect is restored by one conversion kernel at the conv -> dense boundary.

``ConvNetEngine`` covers ``(conv | max_pooling)* dense+`` - every model of the reference's benchmarks. ``StagedEngine``
chains such units for any other order the configuration accepts (dense layers before convolutions, several conv / dense
alternations): a dense block in the middle hands its activation rows to the next unit's convolutions and receives the
gradient w.r.t. its last pre-activation back from them.
"""
from __future__ import annotations

import torch

from ..ops import conv as cv
from ..ops import elementwise as ew
from ..ops.gemm import _fixed_split, gemm
from .engine import Beside, GpuEngine, _up, on_device_rows


def wgrad_split(bf16: bool, F: int, ckk: int, rows: int, sms: int) -> dict:
    """How a convolution's weight gradient ([F, ckk], reduced over ``rows`` output pixels) is split: arguments for ``gemm``.

    bf16 tiles: one number of splits per shape, as many as fill the SMs with 128-column tiles (see ``GpuEngine.fixed_order``); the
    tiles are twice as wide, so that they run in one wave (64 x 288 over 401408 pixels in 50 splits: 150 tiles of 128 columns
    111.5 us, 100 of 256 84, the library's 49 splits 73; events around a cold call, which adds about 8).

    tf32: the library splits results of up to an eighth as many tiles as SMs. Up to a quarter it takes clusters of four CTAs, which
    leave many SMs idle: from 400 k-blocks on more splits pay (200 x 1200 over 100352 pixels: 270 -> 188 us; 384 x 900 over 25088: 78 ->
    69; 200 x 1200 over 6272, 196 k-blocks: 28.7 -> 29.7)."""
    tiles = -(-F // 128) * -(-ckk // 128)
    kb = -(-rows // (64 if bf16 else 32))
    if bf16:
        return dict(split_k=max(1, min(kb, -(-sms // tiles))), bn=256 if ckk > 128 else 0, cluster=-1)
    return dict(split_k=sms // tiles) if 4 * tiles <= sms < 8 * tiles and kb >= 400 else {}


class ConvNetEngine:
    """``ConvFront`` + the dense ``GpuEngine``, with the interface the rank runtime uses."""

    def __init__(self, layers: list[dict], *, batch_size: int, tile_dtype: str, loss: str, params: torch.Tensor,
                 grads: torch.Tensor, params_bf16: torch.Tensor | None = None, leaky_relu_exact: bool = True,
                 bias_from_shadow: bool = False, first: bool = True, prev_act=None, final: bool = True):
        # first = False: this unit follows a dense block. Its input arrives as activation rows of that block (not as a
        # batch), and backward also produces the gradient w.r.t. that block's last pre-activation (``prev_act`` is that
        # layer's activation: its derivative is applied from the stored activation, like between two layers).
        self.first, self.prev_act = first, prev_act
        nfront = 0
        while nfront < len(layers) and layers[nfront]["kind"] != "dense":
            nfront += 1
        if nfront == len(layers):
            raise NotImplementedError("a model needs at least one dense layer after its conv/pool layers on the GPU")
        if any(l["kind"] != "dense" for l in layers[nfront:]):
            raise NotImplementedError("conv/pool layers after a dense layer are not supported on the GPU engine")
        self.bf16 = tile_dtype == "bf16"
        self.dev = params.device
        # tf32 weight gradients read dy and the columns in place as MN-major operands (no transposed copies of either);
        # ONO_CONV_TF32_T=1 brings back the K-major operands with their transposed copies
        self.wgrad_t = tile_dtype != "bf16" and __import__("os").environ.get("ONO_CONV_TF32_T", "0") == "1"
        self.B = batch_size
        self.relu_quirk = not leaky_relu_exact
        self.params, self.grads, self.params_bf16 = params, grads, params_bf16
        self.T = torch.bfloat16 if self.bf16 else torch.float32
        off = 0
        self.front = []
        for sp in layers[:nfront]:
            c, h, w = sp["input_dim"]
            d = dict(sp)
            if sp["kind"] == "conv":
                f, _, k = sp["kernel_dim"]
                d.update(C=c, H=h, W=w, F=f, K=k, off=off, n=f * c * k * k + f)
                off += d["n"]
            else:
                d.update(C=c, H=h, W=w, F=c, K=sp["filter_size"], off=off, n=0)
            d["S"], d["P"] = sp["stride"], sp["padding"]
            d["OH"] = (h + 2 * d["P"] - d["K"]) // d["S"] + 1
            d["OW"] = (w + 2 * d["P"] - d["K"]) // d["S"] + 1
            self.front.append(d)
        self.front_params = off
        last = self.front[-1]
        dense_layers = layers[nfront:]
        assert dense_layers[0]["in"] == last["F"] * last["OH"] * last["OW"]
        self.dense = GpuEngine(dense_layers, batch_size=batch_size, tile_dtype=tile_dtype, loss=loss,
                               params=params[off:], grads=grads[off:],
                               params_bf16=None if params_bf16 is None else params_bf16[off:],
                               leaky_relu_exact=leaky_relu_exact, bias_from_shadow=False, input_grad=True, final=final)
        self.dense.fixed_order = self.bf16
        self.sms = torch.cuda.get_device_properties(self.dev).multi_processor_count
        self.n_params = off + self.dense.n_params
        self.loss_sum, self.correct, self.status = self.dense.loss_sum, self.dense.correct, self.dense.status
        self._alloc()

    # the f32 master is read for the (small) kernel tensors and biases of the front
    needs_f32_params = True

    def _alloc(self):
        B, T, dev = self.B, self.T, self.dev
        z = lambda r, c, dt=T: torch.zeros(r, c, device=dev, dtype=dt)
        for j, d in enumerate(self.front):
            Mout = B * d["OH"] * d["OW"]
            d["y"] = z(Mout, _up(d["F"]))
            d["dy"] = z(Mout, _up(d["F"]))
            if d["kind"] == "conv":
                ckk = d["C"] * d["K"] * d["K"]
                d["ckk"] = ckk
                # first layer with one input channel: direct CUDA-core kernels (K = k*k is too short for the tensor cores)
                d["direct"] = j == 0 and self.first and d["C"] == 1 and d["K"] <= 5 and d["F"] <= 128
                if d["direct"]:
                    continue
                d["cols"] = z(Mout, _up(ckk))
                d["gk_tmp"] = z(d["F"], _up(ckk), torch.float32)
                if self.wgrad_t:
                    d["colsT"] = z(ckk, _up(Mout))
                    d["dyT"] = z(d["F"], _up(Mout))
                d["kt"] = z(ckk, _up(d["F"]))                         # K^T for dgrad
                # the kernel tensor as a GEMM operand: rows in (ky, kx, c) order, rebuilt at every refresh
                d["kop"] = z(d["F"], _up(ckk))[:, :ckk]
            else:
                d["arg"] = torch.zeros(Mout, d["C"], device=dev, dtype=torch.int32)
        c0 = self.front[0]
        self.xflat = z(B, _up(c0["C"] * c0["H"] * c0["W"]))   # the batch as rows, in the tile dtype
        # pixel-major input batch; one channel in rows without padding is pixel-major as it stands
        self.x0_in_place = c0.get("direct", False) and self.xflat.shape[1] == c0["H"] * c0["W"]
        self.x0 = self.xflat.view(-1, 1) if self.x0_in_place else z(B * c0["H"] * c0["W"], _up(c0["C"]))
        self.in_stub = None
        if not self.first:
            # stands in for "the layer below the first one": its output is this unit's input, its gradient buffer receives
            # d(loss)/d(pre-activation of the dense layer that produced the input), pixel-major
            self.dx0 = z(B * c0["H"] * c0["W"], _up(c0["C"]))
            self.in_stub = {"kind": "conv", "y": self.x0, "dy": self.dx0, "act": self.prev_act, "direct": True}
        for j, d in enumerate(self.front):
            prev = self.front[j - 1] if j > 0 else self.in_stub
            if d["kind"] != "conv" or d.get("direct"):
                continue
            g = cv.geom(B, d["C"], d["H"], d["W"], d["K"], d["S"], d["P"])
            # columns and product in one kernel where it takes the sizes and, for the rows there are, pays: see _gathers
            d["gather"] = not self.wgrad_t and cv.fprop_fits(g, d["F"], self.x0 if j == 0 else self.front[j - 1]["y"], d["kop"], d["y"], d["cols"])
            if prev is None:
                continue
            # product and fold in one kernel where it takes the sizes and is the faster form; else the column gradient goes through memory
            d["fold"] = (not self.wgrad_t and cv.dgrad_fits(g, d["F"], d["dy"], d["kt"], prev["dy"], prev["y"])
                         and cv.dgrad_pays(g, d["F"], self.T))
            if not d["fold"]:
                d["dcols"] = z(B * d["OH"] * d["OW"], _up(d["ckk"]))

    def set_side(self, stream) -> None:
        self.dense.set_side(stream)

    def set_report(self, host) -> None:
        self.dense.set_report(host)

    def _k_view(self, d):
        return self.params[d["off"]:d["off"] + d["F"] * d["ckk"]].view(d["F"], d["ckk"])

    def _kb_view(self, d):
        return self.params[d["off"] + d["F"] * d["ckk"]:d["off"] + d["n"]]

    def refresh(self, stream=None) -> int:
        n = 0
        for d in self.front:
            if d["kind"] != "conv" or d.get("direct"):
                continue
            cv.kernel_to_operand(d["F"], d["C"], d["K"], self._k_view(d), d["kop"],
                                 d["kt"][:, :d["F"]] if not self.bf16 or d.get("fold") else None, stream=stream)
            n += 1
        return n + self.dense.refresh(stream)

    def _gathers(self, d, g) -> bool:
        """``d["gather"]``, but not where two kernels are faster, nor where the fixed order splits the reduction (few rows under a long one)."""
        return (d["gather"] and cv.fprop_pays(g, d["F"], self.T)
                and (not self.bf16 or _fixed_split(g.B * g.OH * g.OW, d["F"], d["ckk"], 2, False, self.sms) == 1))

    def _pool_flat(self, g) -> bool:
        """Whether a pooling layer that the dense layers follow runs together with the change to their rows."""
        return not self.wgrad_t and cv.pool_flat_fits(g, self.T)

    def _act(self, d):
        a = d.get("act")
        return (a[0], a[1]) if a else (None, 0.0)

    def batch_job(self, x: torch.Tensor, nrows: int) -> dict:
        """The f32 batch as rows in the tile dtype: arguments for ``ew.rows``."""
        return dict(src=x, n_rows=nrows, **{"dst_bf16" if self.bf16 else "dst": self.xflat})

    def _pixels(self, x: torch.Tensor, nrows: int) -> torch.Tensor | None:
        """The batch as the first layer reads it, where it lies: one channel, f32, rows without a gap."""
        c0 = self.front[0]
        width = c0["C"] * c0["H"] * c0["W"]
        if self.bf16 or not self.x0_in_place or not on_device_rows(x, nrows, width) or x.stride(0) != width:
            return None
        return x[:nrows].view(-1, 1)

    def forward_front(self, rows: torch.Tensor, nrows: int, stream=None, x0: torch.Tensor | None = None) -> int:
        """``rows``: the batch (``xflat``, first unit) or the activation rows of the dense block below, in the tile dtype; ``x0``: its pixels
        where they need no copy."""
        n = 0
        c0 = self.front[0]
        xin = c0["C"] * c0["H"] * c0["W"]
        if x0 is None and not self.x0_in_place:
            cv.nchw_flat(nrows, c0["C"], c0["H"] * c0["W"], False, self.x0, rows[:, :xin], stream=stream)
            n += 1
        cur = self.x0 if x0 is None else x0
        last, de = self.front[-1], self.dense
        for d in self.front:
            Mout = nrows * d["OH"] * d["OW"]
            g = cv.geom(nrows, d["C"], d["H"], d["W"], d["K"], d["S"], d["P"])
            act, ap = self._act(d)
            if d["kind"] == "conv" and d.get("direct"):
                cv.conv1_fwd(g, d["F"], cur, self._k_view(d), self._kb_view(d), d["y"], act=act, act_param=ap, stream=stream)
                n += 1
            elif d["kind"] == "conv" and self._gathers(d, g):
                cv.fprop(g, d["F"], cur, d["kop"], d["y"], cols=d["cols"], bias=self._kb_view(d), act=act, act_param=ap, status=self.status,
                         stream=stream)
                n += 1
            elif d["kind"] == "conv":
                cv.im2col(g, cur, d["cols"], d["colsT"] if self.wgrad_t else None, stream=stream)
                kw = dict(bias=self._kb_view(d), act=act, act_param=ap, fixed_order=self.bf16, status=self.status, stream=stream)
                if self.bf16:
                    kw["out_bf16"] = d["y"][:Mout, :d["F"]]
                else:
                    kw["out"] = d["y"][:Mout, :d["F"]]
                gemm(d["cols"][:Mout, :d["ckk"]], d["kop"], **kw)
                n += 2
            elif d is last and self._pool_flat(g):
                cv.pool_flat_fwd(g, cur, d["y"], d["arg"], de.a[0], act=act, act_param=ap, stream=stream)
                return n + 1
            else:
                cv.pool_fwd(g, cur, d["y"], d["arg"], act=act, act_param=ap, stream=stream)
                n += 1
            cur = d["y"]
        cv.nchw_flat(nrows, last["F"], last["OH"] * last["OW"], True, last["y"], de.a[0], stream=stream)
        return n + 1

    def backward_front(self, nrows: int, accumulate: bool, stream=None, grad_rows: torch.Tensor | None = None,
                       bias_jobs: list | None = None, x0: torch.Tensor | None = None, beside: bool = False) -> int:
        """``grad_rows`` (units after the first): where the gradient w.r.t. the last pre-activation of the dense block below goes, as
        rows in the tile dtype. ``bias_jobs``: bias gradients collected so far, summed beside the first layer's weight gradient (None:
        each layer's on its own). ``x0``: the pixels that forward had. ``beside``: something of this step runs on the second
        stream already."""
        n = 0
        de = self.dense
        last = self.front[-1]
        act, ap = self._act(last) if last["kind"] == "conv" else (None, 0.0)
        want_t = self.wgrad_t and last["kind"] == "conv" and not last.get("direct")
        flat = last["kind"] != "conv" and self._pool_flat(cv.geom(nrows, last["C"], last["H"], last["W"], last["K"], last["S"], last["P"]))
        if not flat:
            cv.nchw_flat(nrows, last["F"], last["OH"] * last["OW"], False, last["dy"], de.d[0],
                         out_t=last["dyT"] if want_t else None, aux=last["y"], dact=act, dact_param=ap,
                         relu_quirk=self.relu_quirk, stream=stream)
            n += 1
        par = Beside(stream, de.side)
        par.used = beside

        def bias_sums(j):
            """At the first layer every delta exists: the collected bias gradients at once, beside its weight gradient."""
            if j > 0 or not bias_jobs:
                return 0
            par.mark(True)
            return ew.colsum_jobs(bias_jobs, stream=par.on())

        for j in range(len(self.front) - 1, -1, -1):
            d = self.front[j]
            prev = self.front[j - 1] if j > 0 else self.in_stub
            Mout = nrows * d["OH"] * d["OW"]
            g = cv.geom(nrows, d["C"], d["H"], d["W"], d["K"], d["S"], d["P"])
            pact, pap = (self._act(prev) if (prev is not None and prev["kind"] == "conv") else (None, 0.0))
            prev_t = prev is not None and prev["kind"] == "conv" and self.wgrad_t and not prev.get("direct")
            if d["kind"] == "conv" and d.get("direct"):
                F, ckk = d["F"], d["ckk"]
                n += bias_sums(j)
                cv.conv1_wgrad(g, F, self.x0 if x0 is None else x0, d["dy"], self.grads[d["off"]:d["off"] + F * ckk],
                               self.grads[d["off"] + F * ckk:d["off"] + d["n"]], beta=1.0 if accumulate else 0.0, stream=stream)
                n += 1
            elif d["kind"] == "conv":
                F, ckk = d["F"], d["ckk"]
                dy = d["dy"][:Mout, :F]
                gb, bbeta = self.grads[d["off"] + F * ckk:d["off"] + d["n"]], 1.0 if accumulate else 0.0
                if bias_jobs is not None:
                    bias_jobs.append((dy, gb, bbeta))
                    n += bias_sums(j)
                else:
                    ew.colsum(dy, gb, beta=bbeta, stream=stream)
                    n += 1
                par.mark(prev is not None)
                if prev is not None and d["fold"]:
                    cv.dgrad(g, F, dy, d["kt"], prev["dy"], aux=prev["y"], dact=pact, dact_param=pap, relu_quirk=self.relu_quirk,
                             status=self.status, stream=stream)
                    n += 1
                elif prev is not None:
                    if self.bf16:
                        gemm(dy, d["kop"], b_mn_major=True, out_bf16=d["dcols"][:Mout, :ckk], fixed_order=True, status=self.status,
                             stream=stream)
                    else:
                        gemm(dy, d["kt"][:, :F], out=d["dcols"][:Mout, :ckk], status=self.status, stream=stream)
                    cv.col2im(g, d["dcols"], prev["dy"], prev["dyT"] if prev_t else None, aux=prev["y"], dact=pact,
                              dact_param=pap, relu_quirk=self.relu_quirk, stream=stream)
                    n += 2
                # weight gradient: K = every output pixel of the batch, tiny output
                tmp, ws = d["gk_tmp"], par.on()
                if not self.wgrad_t:
                    gemm(dy, d["cols"][:Mout, :ckk], a_mn_major=True, b_mn_major=True, out=tmp[:, :ckk], status=self.status,
                         stream=ws, **wgrad_split(self.bf16, F, ckk, Mout, self.sms))
                else:
                    gemm(d["dyT"][:, :Mout], d["colsT"][:, :Mout], out=tmp[:, :ckk], status=self.status, stream=ws,
                         **wgrad_split(False, F, ckk, Mout, self.sms))
                gk = self.grads[d["off"]:d["off"] + F * ckk]
                cv.operand_grad_to_kernel(F, d["C"], d["K"], tmp[:, :ckk], gk, beta=1.0 if accumulate else 0.0, stream=ws)
                n += 3      # split GEMM + finishing pass, permutation
            else:
                n += bias_sums(j)
                if prev is None:
                    continue
                act, ap = self._act(d)
                if d is last and flat:
                    cv.pool_flat_bwd(g, de.d[0], d["y"], d["arg"], prev["dy"], act=act, act_param=ap, aux=prev["y"], dact=pact, dact_param=pap,
                                     relu_quirk=self.relu_quirk, stream=stream)
                    n += 1
                    continue
                cv.pool_bwd(g, d["dy"], d["y"], d["arg"], prev["dy"], prev["dyT"] if prev_t else None, act=act, act_param=ap,
                            aux=prev["y"], dact=pact, dact_param=pap, relu_quirk=self.relu_quirk, stream=stream)
                n += 1
        par.join()
        if self.in_stub is not None:
            c0 = self.front[0]
            xin = c0["C"] * c0["H"] * c0["W"]
            cv.nchw_flat(nrows, c0["C"], c0["H"] * c0["W"], True, self.dx0, grad_rows[:, :xin], stream=stream)
            n += 1
        return n

    def step(self, x, y, nrows, idx=None, accumulate=False, stream=None, after_layer=None, zero_loss=False) -> int:
        if idx is not None:
            raise NotImplementedError("index gather is done by the batch feeder for conv models")
        de = self.dense
        labels = dict(src=y, n_rows=nrows, dst=de.ybuf)
        t = de.small_from()
        if t is not None:
            x0, y_here = self._pixels(x, nrows), on_device_rows(y, nrows, de.plans[-1].out_features)
            jobs = ([] if x0 is not None else [self.batch_job(x, nrows)]) + ([] if y_here else [labels])
            n = ew.rows_jobs(jobs, stream=stream)
            n += self.forward_front(self.xflat, nrows, stream, x0) + de.forward(nrows, stream, upto=t) + 2
            s = de.small_rows(de.a[t], y if y_here else de.ybuf, nrows, stream, zero_loss)
            bias_jobs: list = []
            if t:
                n += de.backward(nrows, accumulate, stream, bias_jobs=bias_jobs, tail=s)
                return n + self.backward_front(nrows, accumulate, stream, bias_jobs=bias_jobs, x0=x0)
            grads = Beside(stream, de.side)
            grads.mark(True)
            de.small_grads(s, accumulate, grads.on())
            return n + self.backward_front(nrows, accumulate, stream, bias_jobs=bias_jobs, x0=x0, beside=grads.used)
        n = ew.rows_jobs([self.batch_job(x, nrows), labels], zero=self.loss_sum if zero_loss else None, stream=stream)
        n += self.forward_front(self.xflat, nrows, stream)
        n += de.forward(nrows, stream)
        n += de.loss_backward(nrows, stream)
        bias_jobs = []
        n += de.backward(nrows, accumulate, stream, bias_jobs=bias_jobs)
        return n + self.backward_front(nrows, accumulate, stream, bias_jobs=bias_jobs)


def _units(layers: list[dict]) -> list[tuple[list[dict], list[dict]]]:
    """Split a layer list into (conv/pool run, dense run) units; a model must end with a dense layer."""
    out, i = [], 0
    while i < len(layers):
        front, dense = [], []
        while i < len(layers) and layers[i]["kind"] != "dense":
            front.append(layers[i]); i += 1
        while i < len(layers) and layers[i]["kind"] == "dense":
            dense.append(layers[i]); i += 1
        if not dense:
            raise NotImplementedError("a model needs a dense layer after its last conv/pool layer on the GPU")
        out.append((front, dense))
    return out


class StagedEngine:
    """Units of ``(conv | pool)* dense+`` chained in any order the model asks for (machine_learning/src/arch/layer.rs:10-19
    puts no order on the layer kinds). Every unit but the last ends in a dense block whose activation rows feed the next
    unit's convolutions."""

    needs_f32_params = True

    def __init__(self, layers: list[dict], *, batch_size: int, tile_dtype: str, loss: str, params: torch.Tensor,
                 grads: torch.Tensor, params_bf16: torch.Tensor | None = None, leaky_relu_exact: bool = True,
                 bias_from_shadow: bool = False):
        units = _units(layers)
        self.B, self.max_ctas = batch_size, 0
        self.units, off = [], 0
        kw = dict(batch_size=batch_size, tile_dtype=tile_dtype, loss=loss, leaky_relu_exact=leaky_relu_exact)
        for k, (front, dense) in enumerate(units):
            final = k == len(units) - 1
            pb = None if params_bf16 is None else params_bf16[off:]
            if front:
                prev_act = units[k - 1][1][-1].get("act") if k > 0 else None
                u = ConvNetEngine(front + dense, params=params[off:], grads=grads[off:], params_bf16=pb, first=k == 0,
                                  prev_act=prev_act, final=final, **kw)
            else:           # only the first unit can be dense-only
                u = GpuEngine(dense, params=params[off:], grads=grads[off:], params_bf16=pb, bias_from_shadow=False, final=final,
                              **kw)
                u.fixed_order = u.bf16
            off += u.n_params
            self.units.append(u)
        self.n_params = off
        last = self._dense(self.units[-1])
        self.loss_sum, self.correct, self.status = last.loss_sum, last.correct, last.status
        for u in self.units:        # one status word for every GEMM of the model
            u.status = self.status
            self._dense(u).small = None
            if isinstance(u, ConvNetEngine):
                u.dense.status = self.status

    @staticmethod
    def _dense(u) -> GpuEngine:
        return u.dense if isinstance(u, ConvNetEngine) else u

    def set_side(self, stream) -> None:
        for u in self.units:
            u.set_side(stream)

    def set_report(self, host) -> None:
        self._dense(self.units[-1]).set_report(host)

    def refresh(self, stream=None) -> int:
        return sum(u.refresh(stream) for u in self.units)

    def step(self, x, y, nrows, idx=None, accumulate=False, stream=None, after_layer=None, zero_loss=False) -> int:
        if idx is not None:
            raise NotImplementedError("index gather is done by the batch feeder for conv models")
        last = self._dense(self.units[-1])
        n = ew.rows_jobs([self.units[0].batch_job(x, nrows), dict(src=y, n_rows=nrows, dst=last.ybuf)],
                         zero=self.loss_sum if zero_loss else None, stream=stream)
        rows_in = None
        for k, u in enumerate(self.units):
            if isinstance(u, ConvNetEngine):
                n += u.forward_front(u.xflat if k == 0 else rows_in, nrows, stream)
                n += u.dense.forward(nrows, stream)
            else:
                n += u.forward(nrows, stream)
            rows_in = self._dense(u).out_act
        n += last.loss_backward(nrows, stream)
        for k in range(len(self.units) - 1, -1, -1):
            u = self.units[k]
            if isinstance(u, ConvNetEngine):
                n += u.dense.backward(nrows, accumulate, stream)
                below = self._dense(self.units[k - 1]) if k > 0 else None
                n += u.backward_front(nrows, accumulate, stream, grad_rows=None if below is None else below.d[-1])
            else:
                n += u.backward(nrows, accumulate, stream)
        return n


def make_engine(layers: list[dict], **kw):
    """The engine for a layer list: dense-only, one conv/pool front followed by dense layers, or chained units."""
    if all(l["kind"] == "dense" for l in layers):
        return GpuEngine(layers, **kw)
    if len(_units(layers)) == 1:
        return ConvNetEngine(layers, **kw)
    return StagedEngine(layers, **kw)
