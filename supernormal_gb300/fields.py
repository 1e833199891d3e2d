"""SDF field modules: drop-in for models/fields.py on the sm_103a kernels.

``SDFNetwork`` keeps the reference constructor (models/fields.py:8-70), its
geometric initialisation (same torch RNG call sequence), its state_dict keys
(``encoding.params``, ``lin{l}.bias``, ``lin{l}.weight_g``,
``lin{l}.weight_v``), ``bindwidth`` / ``increase_bandwidth`` and the
``forward / sdf / gradient`` methods.  The hash-grid encoding (the
``tcnn.Encoding`` of models/fields.py:26) and the MLP run fused in one
kernel with a hand-written backward; the MLP shape the kernels cover is the
one SuperNormal ships: one hidden layer of 64 with input concatenation.
"""
from __future__ import annotations

import ctypes as C
import threading
from typing import Optional

import numpy as np
import torch
import torch.nn as nn
from torch import Tensor

from ._lib import SN_STATUS_TIMEOUT, GridDesc, MlpDesc, WeightNormLayer, call, lib, stream_handle

__all__ = ["HashGridEncoding", "WeightNormLinear", "SDFNetwork", "SingleVarianceNetwork",
           "grid_desc"]


def grid_desc(n_levels: int, n_features_per_level: int, log2_hashmap_size: int,
              base_resolution: int, per_level_scale: float) -> GridDesc:
    """tcnn GridEncoding level geometry (offsets, resolutions, scales)."""
    d = GridDesc()
    call("sn_grid_desc_init", C.byref(d), int(n_levels), int(n_features_per_level),
         int(log2_hashmap_size), int(base_resolution), float(per_level_scale))
    return d


def _need_cuda(t: Tensor) -> None:
    if not t.is_cuda:
        raise NotImplementedError("supernormal_gb300 fields run on CUDA tensors only")


class HashGridEncoding(nn.Module):
    """Multi-resolution hash encoding with tcnn's parameter layout; parameter
    ``params`` is the flat table (offsets[L] * F floats), initialised
    uniform(-1e-4, 1e-4) like tcnn's GridEncoding."""

    def __init__(self, n_input_dims: int, encoding_config: dict, seed: int = 1337,
                 dtype=torch.float32):
        super().__init__()
        otype = encoding_config.get("otype", "HashGrid")
        if otype not in ("HashGrid", "Grid") or encoding_config.get("type", "Hash") != "Hash":
            raise NotImplementedError(f"encoding otype {otype!r} is not supported (HashGrid only)")
        if n_input_dims != 3:
            raise NotImplementedError("only 3-D inputs are supported")
        if encoding_config.get("interpolation", "Linear") != "Linear":
            raise NotImplementedError("only linear interpolation is supported")
        self.n_input_dims = n_input_dims
        self.n_levels = int(encoding_config.get("n_levels", 16))
        self.n_features_per_level = int(encoding_config.get("n_features_per_level", 2))
        self.log2_hashmap_size = int(encoding_config.get("log2_hashmap_size", 19))
        self.base_resolution = int(encoding_config.get("base_resolution", 16))
        self.per_level_scale = float(encoding_config.get("per_level_scale", 2.0))
        self.desc = grid_desc(self.n_levels, self.n_features_per_level, self.log2_hashmap_size,
                              self.base_resolution, self.per_level_scale)
        self.n_output_dims = self.n_levels * self.n_features_per_level
        n_params = int(self.desc.offsets[self.n_levels]) * self.n_features_per_level
        gen = torch.Generator().manual_seed(int(seed))
        init = (torch.rand(n_params, generator=gen, dtype=torch.float64) * 2.0 - 1.0) * 1e-4
        self.params = nn.Parameter(init.to(dtype))

    @property
    def n_params(self) -> int:
        return self.params.numel()

    def level_offsets(self) -> np.ndarray:
        return np.array(self.desc.offsets[: self.n_levels + 1], dtype=np.int64)

    def level_resolutions(self) -> np.ndarray:
        return np.array(self.desc.resolutions[: self.n_levels], dtype=np.int64)

    def level_scales(self) -> np.ndarray:
        return np.array(self.desc.scales[: self.n_levels], dtype=np.float32)

    def forward(self, x: Tensor, active_levels: Optional[int] = None) -> Tensor:
        _need_cuda(x)
        act = self.n_levels if active_levels is None else int(active_levels)
        return _HashGridFn.apply(x, self.params, self, act)


class _HashGridFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x: Tensor, table: Tensor, enc: HashGridEncoding, active: int):
        x = x.contiguous().float()
        out = torch.empty((x.shape[0], enc.n_output_dims), device=x.device, dtype=torch.float32)
        call("sn_hashgrid_fwd", x.shape[0], x, table, C.byref(enc.desc), active, out, stream_handle())
        ctx.save_for_backward(x)
        ctx.enc, ctx.active, ctx.n_table = enc, active, table.numel()
        return out

    @staticmethod
    def backward(ctx, grad_out: Tensor):
        (x,) = ctx.saved_tensors
        gt = None
        if ctx.needs_input_grad[1]:
            gt = torch.zeros(ctx.n_table, device=x.device, dtype=torch.float32)
            call("sn_hashgrid_bwd", x.shape[0], x, grad_out.contiguous().float(),
                 C.byref(ctx.enc.desc), ctx.active, gt, stream_handle())
        if ctx.needs_input_grad[0]:
            raise NotImplementedError("d(encoding)/dx alone is not exposed; use SDFNetwork.gradient")
        return None, gt, None, None


class _WeightNorm(torch.autograd.Function):
    """w = g * v / ||v|| per output row (torch.nn.utils.weight_norm, dim=0)."""

    @staticmethod
    def forward(ctx, v: Tensor, g: Tensor):
        v = v.contiguous().float()
        g = g.contiguous().float()
        rows, cols = v.shape
        w = torch.empty_like(v)
        norms = torch.empty((rows,), device=v.device, dtype=torch.float32)
        call("sn_weightnorm_fwd", rows, cols, v, g, w, norms, stream_handle())
        ctx.save_for_backward(v, g, norms)
        return w

    @staticmethod
    def backward(ctx, gw: Tensor):
        v, g, norms = ctx.saved_tensors
        rows, cols = v.shape
        gv = torch.empty_like(v)
        gg = torch.empty((rows,), device=v.device, dtype=torch.float32)
        call("sn_weightnorm_bwd", rows, cols, v, g, norms, gw.contiguous().float(), gv, gg,
             stream_handle())
        return gv, gg.reshape(g.shape)


class WeightNormLinear(nn.Module):
    """Linear layer with the parameters torch's weight_norm registers
    (``weight_g`` (out, 1), ``weight_v`` (out, in), ``bias``)."""

    def __init__(self, lin: nn.Linear, weight_norm: bool = True):
        super().__init__()
        self.use_wn = weight_norm
        w = lin.weight.detach().clone()
        if weight_norm:
            self.weight_g = nn.Parameter(torch.linalg.vector_norm(w, dim=1, keepdim=True))
            self.weight_v = nn.Parameter(w)
        else:
            self.weight = nn.Parameter(w)
        self.bias = nn.Parameter(lin.bias.detach().clone())
        self.in_features, self.out_features = lin.in_features, lin.out_features

    def effective_weight(self) -> Tensor:
        if not self.use_wn:
            return self.weight
        if self.weight_v.is_cuda:
            return _WeightNorm.apply(self.weight_v, self.weight_g)
        return self.weight_g * self.weight_v / torch.linalg.vector_norm(self.weight_v, dim=1,
                                                                       keepdim=True)


class _FieldFn(torch.autograd.Function):
    """Fused encoding + MLP; backward recomputes activations (no stored hidden state)."""

    @staticmethod
    def forward(ctx, x, table, w0, b0, w1, b1, net: "SDFNetwork", out_cols: int):
        x = x.contiguous().float()
        active = net.active_levels()
        desc = net._mlp_desc(w0, b0, w1, b1)
        out = torch.empty((x.shape[0], out_cols), device=x.device, dtype=torch.float32)
        call("sn_field_fwd", x.shape[0], None, x, table, C.byref(net.encoding.desc), active,
             C.byref(desc), out_cols, out, stream_handle())
        ctx.save_for_backward(x, table, w0, b0, w1, b1)
        ctx.net, ctx.out_cols, ctx.active = net, out_cols, active
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, table, w0, b0, w1, b1 = ctx.saved_tensors
        net = ctx.net
        dev = x.device
        need = ctx.needs_input_grad
        g_table = torch.zeros_like(table) if need[1] else None
        g_w0 = torch.zeros_like(w0) if need[2] else None
        g_b0 = torch.zeros_like(b0) if need[3] else None
        g_w1 = torch.zeros_like(w1) if need[4] else None
        g_b1 = torch.zeros_like(b1) if need[5] else None
        g_x = torch.empty_like(x) if need[0] else None
        desc = net._mlp_desc(w0, b0, w1, b1)
        call("sn_field_bwd", x.shape[0], None, x, grad_out.contiguous().float(), ctx.out_cols, table,
             C.byref(net.encoding.desc), ctx.active, C.byref(desc), g_table, g_w0, g_b0, g_w1, g_b1,
             g_x, stream_handle())
        return g_x, g_table, g_w0, g_b0, g_w1, g_b1, None, None


class _FieldGradFn(torch.autograd.Function):
    """(sdf, d sdf/dx) in one kernel; backward is the hand-written second-order
    adjoint (the double backward of models/fields.py:107-119 with create_graph)."""

    @staticmethod
    def forward(ctx, x, table, w0, b0, w1, b1, net: "SDFNetwork"):
        x = x.contiguous().float()
        active = net.active_levels()
        desc = net._mlp_desc(w0, b0, w1, b1)
        sdf = torch.empty((x.shape[0], 1), device=x.device, dtype=torch.float32)
        grad = torch.empty((x.shape[0], 3), device=x.device, dtype=torch.float32)
        call("sn_field_grad_fwd", x.shape[0], None, x, table, C.byref(net.encoding.desc), active,
             C.byref(desc), sdf, grad, stream_handle())
        ctx.save_for_backward(x, table, w0, b0, w1, b1)
        ctx.net, ctx.active = net, active
        return sdf, grad

    @staticmethod
    def backward(ctx, g_sdf, g_grad):
        x, table, w0, b0, w1, b1 = ctx.saved_tensors
        if ctx.needs_input_grad[0]:
            raise NotImplementedError("d^2 sdf / dx^2 (the Hessian) is not implemented")
        need = ctx.needs_input_grad
        g_table = torch.zeros_like(table) if need[1] else None
        g_w0 = torch.zeros_like(w0) if need[2] else None
        g_b0 = torch.zeros_like(b0) if need[3] else None
        g_w1 = torch.zeros_like(w1) if need[4] else None
        g_b1 = torch.zeros_like(b1) if need[5] else None
        g_grad = torch.zeros((x.shape[0], 3), device=x.device) if g_grad is None else g_grad.contiguous().float()
        g_sdf = None if g_sdf is None else g_sdf.contiguous().float().reshape(-1)
        desc = ctx.net._mlp_desc(w0, b0, w1, b1)
        call("sn_field_grad_bwd", x.shape[0], None, x, g_grad, g_sdf, table,
             C.byref(ctx.net.encoding.desc), ctx.active, C.byref(desc), g_table, g_w0, g_b0, g_w1,
             g_b1, stream_handle())
        return None, g_table, g_w0, g_b0, g_w1, g_b1, None


class _WeightNormField:
    """The weight-normalised network of a field call: its effective weights
    (one buffer: w0, w1 and the row norms of both) and the descriptors that the
    library takes.  One autograd node then holds what the layers' and the
    field's did (three nodes cost more host time than the kernels take at
    100,000 points)."""

    def __init__(self, net: "SDFNetwork", v0: Tensor, g0: Tensor, b0: Tensor, v1: Tensor, g1: Tensor, b1: Tensor,
                 w: Optional[Tensor] = None, enc: Optional[Tensor] = None):
        (h, din), dout = v0.shape, v1.shape[0]
        if w is None:
            w = torch.empty((h * din + dout * h + h + dout,), device=v0.device, dtype=torch.float32)
        self.w, self.sizes = w, (h, din, dout)
        self.w0 = w.data_ptr()
        self.w1 = self.w0 + 4 * h * din
        self.n0 = self.w1 + 4 * dout * h
        self.n1 = self.n0 + 4 * h
        self.v = (v0.data_ptr(), g0.data_ptr(), v1.data_ptr(), g1.data_ptr())
        self.mlp = C.byref(MlpDesc(din, h, dout, net.beta, net.threshold, self.w0, b0.data_ptr(), self.w1,
                                   b1.data_ptr(), net._kernel_status.data_ptr(), 0,
                                   enc.data_ptr() if enc is not None else None))

    def layers(self, grads=None):
        """The layers' descriptors; grads: (scratch for the weight gradients,
        grad_v0, grad_g0, grad_v1, grad_g1)."""
        h, din, dout = self.sizes
        a = b = ()
        if grads is not None:
            gw, gv0, gg0, gv1, gg1 = (t.data_ptr() for t in grads)
            gw1 = gw + 4 * h * din   # h is even: the sums in double behind it are aligned
            a, b = (gw, gv0, gg0), (gw1, gv1, gg1, gw1 + 4 * dout * h)
        return (C.byref(WeightNormLayer(h, din, self.v[0], self.v[1], self.w0, self.n0, *a)),
                C.byref(WeightNormLayer(dout, h, self.v[2], self.v[3], self.w1, self.n1, *b)))

    def gradients(self, need, table: Tensor, v0, g0, b0, v1, g1, b1):
        """Buffers for the gradients that are needed: (grad_table, grad_b0,
        grad_b1, the layers' five or None).  need: table, v0, g0, b0, v1, g1, b1."""
        h, din, dout = self.sizes
        wn = None
        if need[1] or need[2] or need[4] or need[5]:
            wn = (torch.empty((h * din + 3 * dout * h,), device=v0.device, dtype=torch.float32), torch.empty_like(v0),
                  torch.empty_like(g0), torch.empty_like(v1), torch.empty_like(g1))
        return (torch.empty_like(table) if need[0] else None, torch.empty_like(b0) if need[3] else None,
                torch.empty_like(b1) if need[6] else None, wn)

    @staticmethod
    def returned(need, g_table, g_b0, g_b1, wn):
        """The gradients in the order of the function's inputs."""
        _, gv0, gg0, gv1, gg1 = wn if wn is not None else (None,) * 5
        return (g_table, gv0 if need[1] else None, gg0 if need[2] else None, g_b0,
                gv1 if need[4] else None, gg1 if need[5] else None, g_b1)


def _float(t: Tensor) -> Tensor:
    return t.contiguous().float()


# Bytes of encodings that a network's evaluations keep for their backwards, all that
# still wait for theirs together (16.7 million points at 16 levels); above, the
# backward gathers them again.  The line is the memory alone: at any size the backward
# that reads them is the faster one (500,000 points: 110 + 204 us with them kept, 101 +
# 279 us gathered again).
_KEPT_ENCODING_BYTES = 1 << 31


class _EncodingBudget:
    """What a network's evaluations keep at the moment.  An evaluation's share is
    given back by its backward, or with its graph."""

    def __init__(self):
        self.held, self.lock = 0, threading.RLock()   # (a share may be given back by the collector at any point)

    def __deepcopy__(self, memo):
        return _EncodingBudget()

    def __reduce__(self):
        return _EncodingBudget, ()

    def take(self, nbytes: int) -> Optional["_Share"]:
        with self.lock:
            if not 0 < nbytes <= _KEPT_ENCODING_BYTES - self.held:
                return None
            self.held += nbytes
        return _Share(self, nbytes)


class _Share:
    def __init__(self, budget: _EncodingBudget, nbytes: int):
        self.budget, self.nbytes = budget, nbytes

    def give_back(self) -> None:
        with self.budget.lock:
            self.budget.held -= self.nbytes
            self.nbytes = 0

    __del__ = give_back


class _FieldWnFn(torch.autograd.Function):
    """_FieldFn of a weight-normalised network, the normalisation included; keep:
    a backward may follow, so the encoding is kept for it."""

    @staticmethod
    def forward(ctx, x, table, v0, g0, b0, v1, g1, b1, net: "SDFNetwork", out_cols: int, keep: bool):
        x, v0, g0, v1, g1, b0, b1 = _float(x), _float(v0), _float(g0), _float(v1), _float(g1), b0.contiguous(), b1.contiguous()
        active = net.active_levels()
        n = x.shape[0]
        enc = ctx.share = None
        if keep and net.encoding_cache and any(ctx.needs_input_grad):
            ctx.share = net._encoding_budget().take(8 * active * n)
        if ctx.share is not None:
            enc = torch.empty((2 * active * n,), device=x.device, dtype=torch.float32)
        f = _WeightNormField(net, v0, g0, b0, v1, g1, b1, enc=enc)
        out = torch.empty((n, out_cols), device=x.device, dtype=torch.float32)
        call("sn_field_wn_fwd", n, None, x, table, C.byref(net.encoding.desc), active, f.mlp, *f.layers(),
             out_cols, out, stream_handle())
        ctx.save_for_backward(x, table, v0, g0, b0, v1, g1, b1, f.w, enc)
        ctx.net, ctx.out_cols, ctx.active = net, out_cols, active
        return out

    @staticmethod
    def backward(ctx, grad_out):
        x, table, *params, w, enc = ctx.saved_tensors
        net, need = ctx.net, ctx.needs_input_grad
        f = _WeightNormField(net, *params, w, enc)
        g_table, g_b0, g_b1, wn = f.gradients(need[1:8], table, *params)
        g_x = torch.empty_like(x) if need[0] else None
        call("sn_field_wn_bwd", x.shape[0], x, grad_out.contiguous().float(), ctx.out_cols, table, table.numel(),
             C.byref(net.encoding.desc), ctx.active, f.mlp, *f.layers(wn), g_table, g_b0, g_b1, g_x, stream_handle())
        if ctx.share is not None:
            ctx.share.give_back()
        return g_x, *f.returned(need[1:8], g_table, g_b0, g_b1, wn), None, None, None


class _FieldGradWnFn(torch.autograd.Function):
    """_FieldGradFn of a weight-normalised network, the normalisation included."""

    @staticmethod
    def forward(ctx, x, table, v0, g0, b0, v1, g1, b1, net: "SDFNetwork"):
        x, v0, g0, v1, g1, b0, b1 = _float(x), _float(v0), _float(g0), _float(v1), _float(g1), b0.contiguous(), b1.contiguous()
        active = net.active_levels()
        f = _WeightNormField(net, v0, g0, b0, v1, g1, b1)
        sdf = torch.empty((x.shape[0], 1), device=x.device, dtype=torch.float32)
        grad = torch.empty((x.shape[0], 3), device=x.device, dtype=torch.float32)
        call("sn_field_wn_grad_fwd", x.shape[0], x, table, C.byref(net.encoding.desc), active, f.mlp, *f.layers(), sdf,
             grad, stream_handle())
        ctx.save_for_backward(x, table, v0, g0, b0, v1, g1, b1, f.w)
        ctx.net, ctx.active = net, active
        return sdf, grad

    @staticmethod
    def backward(ctx, g_sdf, g_grad):
        x, table, *params, w = ctx.saved_tensors
        net, need = ctx.net, ctx.needs_input_grad
        if need[0]:
            raise NotImplementedError("d^2 sdf / dx^2 (the Hessian) is not implemented")
        f = _WeightNormField(net, *params, w)
        g_table, g_b0, g_b1, wn = f.gradients(need[1:8], table, *params)
        g_grad = torch.zeros((x.shape[0], 3), device=x.device) if g_grad is None else g_grad.contiguous().float()
        g_sdf = None if g_sdf is None else g_sdf.contiguous().float().reshape(-1)
        call("sn_field_wn_grad_bwd", x.shape[0], x, g_grad, g_sdf, table, table.numel(), C.byref(net.encoding.desc),
             ctx.active, f.mlp, *f.layers(wn), g_table, g_b0, g_b1, stream_handle())
        return None, *f.returned(need[1:8], g_table, g_b0, g_b1, wn), None


class SDFNetwork(nn.Module):
    """SDF MLP over a hash-grid encoding (models/fields.py:7-130)."""

    # differentiable evaluations keep their encoding for the backward (up to 2 GB a
    # network at a time); False: the backward gathers it again
    encoding_cache: bool = True

    def _encoding_budget(self) -> _EncodingBudget:
        return vars(self).setdefault("_kept_encodings", _EncodingBudget())

    def __init__(self, d_in, d_out, d_hidden, n_layers, skip_in=(4,), bias=0.5,
                 geometric_init=True, weight_norm=True, inside_outside=False,
                 encoding_config=None, input_concat=False):
        super().__init__()
        self.input_concat = input_concat
        dims = [d_in] + [d_hidden for _ in range(n_layers)] + [d_out]
        if encoding_config is None:
            raise NotImplementedError("SDFNetwork needs an encoding_config (models/fields.py:37)")
        self.encoding = HashGridEncoding(d_in, encoding_config)
        dims[0] = self.encoding.n_output_dims
        if input_concat:
            dims[0] += d_in
        self.num_layers = len(dims)
        self.skip_in = skip_in
        self.bindwidth = 0
        self.enc_dim = self.encoding.n_output_dims
        self.d_in, self.d_out, self.d_hidden = d_in, d_out, d_hidden
        for l in range(0, self.num_layers - 1):
            out_dim = dims[l + 1] - dims[0] if l + 1 in self.skip_in else dims[l + 1]
            lin = nn.Linear(dims[l], out_dim)
            if geometric_init:
                if l == self.num_layers - 2:
                    if not inside_outside:
                        torch.nn.init.normal_(lin.weight, mean=np.sqrt(np.pi) / np.sqrt(dims[l]), std=0.0001)
                        torch.nn.init.constant_(lin.bias, -bias)
                    else:
                        torch.nn.init.normal_(lin.weight, mean=-np.sqrt(np.pi) / np.sqrt(dims[l]), std=0.0001)
                        torch.nn.init.constant_(lin.bias, bias)
                elif l == 0:
                    torch.nn.init.constant_(lin.bias, 0.0)
                    torch.nn.init.constant_(lin.weight[:, 3:], 0.0)
                    torch.nn.init.normal_(lin.weight[:, :3], 0.0, np.sqrt(2) / np.sqrt(out_dim))
                elif l in self.skip_in:
                    torch.nn.init.constant_(lin.bias, 0.0)
                    torch.nn.init.normal_(lin.weight, 0.0, np.sqrt(2) / np.sqrt(out_dim))
                    torch.nn.init.constant_(lin.weight[:, -(dims[0] - 3):], 0.0)
                else:
                    torch.nn.init.constant_(lin.bias, 0.0)
                    torch.nn.init.normal_(lin.weight, 0.0, np.sqrt(2) / np.sqrt(out_dim))
            setattr(self, "lin" + str(l), WeightNormLinear(lin, weight_norm))
        self.beta, self.threshold = 100.0, 20.0
        # device status word of the tensor-core field kernels (not in the state_dict)
        self.register_buffer("_kernel_status", torch.zeros(1, dtype=torch.int32), persistent=False)
        self._supported = (n_layers == 1 and d_hidden == 64 and input_concat and d_in == 3
                           and self.encoding.n_features_per_level == 2
                           and self.encoding.n_levels <= 16 and 1 <= d_out <= 16)

    def _check(self, x: Tensor) -> None:
        _need_cuda(x)
        if not self._supported:
            raise NotImplementedError(
                "the fused field kernels cover SDFNetwork(d_in=3, d_hidden=64, n_layers=1, "
                "input_concat=True, d_out<=16) over a HashGrid with 2 features and <=16 levels")

    def increase_bandwidth(self):
        self.bindwidth += 1

    def active_levels(self) -> int:
        # enc_mask[bindwidth*2:] = 0 with 2 features per level (models/fields.py:81-83)
        return max(0, min(self.bindwidth, self.encoding.n_levels))

    def _mlp_desc(self, w0, b0, w1, b1) -> MlpDesc:
        d = MlpDesc()
        d.d_in = w0.shape[1]
        d.d_hidden = w0.shape[0]
        d.d_out = w1.shape[0]
        d.beta = self.beta
        d.threshold = self.threshold
        d.w0, d.b0, d.w1, d.b1 = w0.data_ptr(), b0.data_ptr(), w1.data_ptr(), b1.data_ptr()
        d.status = self._kernel_status.data_ptr()
        return d

    def check_status(self) -> None:
        """Raise if a field kernel reported a failed bounded wait (host sync)."""
        if int(self._kernel_status.item()) & SN_STATUS_TIMEOUT:
            raise RuntimeError("a tensor-core field kernel timed out waiting for its MMAs")

    def mlp_tensors(self):
        return (self.lin0.effective_weight(), self.lin0.bias, self.lin1.effective_weight(),
                self.lin1.bias)

    def _weight_norm_params(self):
        """(v0, g0, b0, v1, g1, b1) if both layers are this module's own
        weight-normalised ones on a GPU, else None (their effective weights are
        then asked for one by one).  A replaced ``mlp_tensors`` or
        ``effective_weight``, of a subclass, a class or an instance, is asked."""
        cls = type(self)
        if (cls.mlp_tensors, cls._mlp_desc) != _NETWORK_METHODS or not vars(self).keys().isdisjoint(_NETWORK_NAMES):
            return None
        out = []
        for lin in (self.lin0, self.lin1):
            if (type(lin) is not WeightNormLinear or not lin.use_wn or "effective_weight" in vars(lin)
                    or WeightNormLinear.effective_weight is not _EFFECTIVE_WEIGHT):
                return None
            p = lin._parameters
            v, g, b = p.get("weight_v"), p.get("weight_g"), p.get("bias")
            if v is None or g is None or b is None or not v.is_cuda:
                return None
            out += (v, g, b)
        return out

    def _field(self, x: Tensor, out_cols: int) -> Tensor:
        self._check(x)
        wn = self._weight_norm_params()
        if wn is not None:
            return _FieldWnFn.apply(x, self.encoding.params, *wn, self, out_cols, torch.is_grad_enabled())
        w0, b0, w1, b1 = self.mlp_tensors()
        return _FieldFn.apply(x, self.encoding.params, w0.contiguous(), b0.contiguous(),
                              w1.contiguous(), b1.contiguous(), self, out_cols)

    def forward(self, inputs: Tensor) -> Tensor:
        return self._field(inputs, self.d_out)

    def sdf(self, x: Tensor) -> Tensor:
        return self._field(x, 1)

    @torch.no_grad()
    def sdf_raw(self, x: Tensor, count: Optional[Tensor] = None) -> Tensor:
        """No-grad sdf (n, 1) of a capacity buffer x; count (device int32) bounds
        the rows evaluated, so no host synchronisation is needed."""
        self._check(x)
        out = torch.empty((x.shape[0], 1), device=x.device, dtype=torch.float32)
        wn = self._weight_norm_params()
        if wn is not None:
            v0, g0, b0, v1, g1, b1 = wn
            v0, g0, v1, g1, b0, b1 = _float(v0), _float(g0), _float(v1), _float(g1), b0.contiguous(), b1.contiguous()
            f = _WeightNormField(self, v0, g0, b0, v1, g1, b1)
            call("sn_field_wn_fwd", x.shape[0], count, x.contiguous(), self.encoding.params,
                 C.byref(self.encoding.desc), self.active_levels(), f.mlp, *f.layers(), 1, out, stream_handle())
            return out
        w0, b0, w1, b1 = (t.detach().contiguous() for t in self.mlp_tensors())
        desc = self._mlp_desc(w0, b0, w1, b1)
        call("sn_field_fwd", x.shape[0], count, x.contiguous(), self.encoding.params.detach(),
             C.byref(self.encoding.desc), self.active_levels(), C.byref(desc), 1, out,
             stream_handle())
        return out

    def sdf_hidden_appearance(self, x: Tensor) -> Tensor:
        return self.forward(x)

    def sdf_and_gradient(self, x: Tensor):
        """(sdf (N, 1), d sdf / d x (N, 3)), both differentiable w.r.t. the parameters."""
        self._check(x)
        wn = self._weight_norm_params()
        if wn is not None:
            return _FieldGradWnFn.apply(x.detach(), self.encoding.params, *wn, self)
        w0, b0, w1, b1 = self.mlp_tensors()
        return _FieldGradFn.apply(x.detach(), self.encoding.params, w0.contiguous(), b0.contiguous(),
                                  w1.contiguous(), b1.contiguous(), self)

    @torch.enable_grad()
    def gradient(self, x: Tensor) -> Tensor:
        """d sdf / d x, (N, 1, 3) (models/fields.py:107-119).  As with the
        reference's create_graph=True, the result is differentiable w.r.t. the
        parameters (second-order adjoint in sn_field_grad_bwd); like the
        reference, x is marked requires_grad."""
        x.requires_grad_(True)
        _, g = self.sdf_and_gradient(x)
        return g.unsqueeze(1)


# what _weight_norm_params stands in for
_NETWORK_METHODS, _NETWORK_NAMES = (SDFNetwork.mlp_tensors, SDFNetwork._mlp_desc), ("mlp_tensors", "_mlp_desc")
_EFFECTIVE_WEIGHT = WeightNormLinear.effective_weight


class SingleVarianceNetwork(nn.Module):
    """inv_s = exp(10 * variance) (models/fields.py:133-139)."""

    def __init__(self, init_val):
        super().__init__()
        self.register_parameter("variance", nn.Parameter(torch.tensor(init_val)))

    def forward(self, x):
        return torch.ones([len(x), 1], device=self.variance.device) * torch.exp(self.variance * 10.0)
