"""Learned warm start for the boundary-inflow inversion.

A 1D-conv encoder plus MLP maps the gauge waveforms of a run (6 gauges x
1125 samples, eta every 0.02 s over 22.5 s) to the 16 spline controls of the
west-edge inflow.  Its prediction seeds the adjoint inversion
(``inversion.invert``); the plain inversion from the reference's cold start
stays the fallback and the measure of the error (the reference has no learned
part; its inversion is
``Examples/inverse/Monai_Valley/Monai_Velley_BC_inversion_spline_lr002/
bc_inversion_train.py:648-768``).

Every training and inference kernel is this project's (``csrc/nn_b200.cu``):
bf16 matrix products with fp32 accumulation on the tcgen05 tensor cores
(convolutions read their patches in place, weight gradients their operands
untransposed), activation adjoints fused into them, Adam.  A pass is one
call into the library.  The network:

=======  ==============================================  ===========
layer    shape                                           parameters
=======  ==============================================  ===========
conv1    6 -> 32 channels, kernel 9, stride 4, pad 4     1,760
conv2    32 -> 64, kernel 8, stride 4, pad 2             16,448
conv3    64 -> 128, kernel 6, stride 2, pad 2            49,280
fc1      128 x 35 -> 96                                  430,176
fc2      96 -> 96                                        9,312
fc3      96 -> 16 (normalised controls)                  1,552
=======  ==============================================  ===========

GELU after every layer but the last; 508,528 parameters (fp32 master copy,
a bf16 copy for the products).  Activations are kept channel-last (NLC), so
a patch of the next convolution is a contiguous slice of them and the last
one flattens to fc1's input without a copy.
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import List, Tuple

import torch

from . import _native as nat

SAMPLES, GAUGES, CONTROLS = 1125, 6, 16
INPUT_SCALE = 100.0                   # eta [m] -> input units (1 cm -> 1)
CONTROL_MEAN, CONTROL_SCALE = 0.0015, 0.0078   # controls ~ U[-0.012, 0.015] m


@dataclass(frozen=True)
class Conv:
    cin: int
    cout: int
    k: int
    stride: int
    pad: int
    lin: int

    @property
    def lout(self) -> int:
        return (self.lin + 2 * self.pad - self.k) // self.stride + 1

    @property
    def kdim(self) -> int:
        return self.k * self.cin

    @property
    def kpad(self) -> int:
        return -(-self.kdim // 16) * 16


@dataclass(frozen=True)
class Dense:
    cin: int
    cout: int

    @property
    def kpad(self) -> int:
        return self.cin


def architecture(samples: int = SAMPLES, gauges: int = GAUGES, controls: int = CONTROLS):
    c1 = Conv(gauges, 32, 9, 4, 4, samples)
    c2 = Conv(32, 64, 8, 4, 2, c1.lout)
    c3 = Conv(64, 128, 6, 2, 2, c2.lout)
    return [c1, c2, c3, Dense(c3.cout * c3.lout, 96), Dense(96, 96), Dense(96, controls)]


def param_layout(layers) -> List[Tuple[int, int, int, int]]:
    """(weight offset, rows, padded cols, bias offset) per layer in the flat
    parameter vector."""
    out, off = [], 0
    for L in layers:
        w = off
        off += L.cout * L.kpad
        b = off
        off += L.cout
        out.append((w, L.cout, L.kpad, b))
    return out, off


class WarmStartNet:
    """The network, its training state and the buffers of one batch size."""

    def __init__(self, device="cuda", seed: int = 0, samples: int = SAMPLES, gauges: int = GAUGES,
                 controls: int = CONTROLS):
        self.dev = torch.device(device)
        self.layers = architecture(samples, gauges, controls)
        self.layout, self.nparams = param_layout(self.layers)
        self.samples, self.gauges, self.controls = samples, gauges, controls
        self.params = torch.zeros(self.nparams, device=self.dev)
        self.grads = torch.zeros_like(self.params)
        self.m = torch.zeros_like(self.params)
        self.v = torch.zeros_like(self.params)
        self.step_count = 0
        self.err = torch.zeros(1, dtype=torch.int32, device=self.dev)
        #: limit of each tensor-core wait of the GEMM kernel (nn_gemm_bf16)
        self.wait_ns = nat.NN_GEMM_WAIT_NS
        g = torch.Generator().manual_seed(seed)
        host = torch.zeros(self.nparams)
        for L, (w, rows, kp, b) in zip(self.layers, self.layout):
            fan_in = L.kdim if isinstance(L, Conv) else L.cin
            bound = 1.0 / math.sqrt(fan_in)
            W = (torch.rand((rows, fan_in), generator=g) * 2 - 1) * bound
            Wp = torch.zeros((rows, kp))
            Wp[:, :fan_in] = W
            host[w:w + rows * kp] = Wp.reshape(-1)
            host[b:b + rows] = (torch.rand(rows, generator=g) * 2 - 1) * bound
        self.params.copy_(host)
        self.params_bf16 = torch.empty(self.nparams, dtype=torch.int16, device=self.dev)
        self._refresh_bf16()
        self._table = (nat.NnLayer * len(self.layers))()
        for t, L, (w, _, kp, b) in zip(self._table, self.layers, self.layout):
            conv = isinstance(L, Conv)
            t.conv, t.cin, t.cout, t.kpad, t.w, t.b = int(conv), L.cin, L.cout, kp, w, b
            if conv:
                t.k, t.stride, t.pad, t.lin, t.lout = L.k, L.stride, L.pad, L.lin, L.lout
        self._cap = 0      # the largest batch that the workspace holds
        self._nb = None    # the last batch

    # ----------------------------------------------------------- helpers
    def weight(self, i):
        w, rows, kp, _ = self.layout[i]
        return self.params[w:w + rows * kp].view(rows, kp)

    def bias(self, i):
        _, rows, _, b = self.layout[i]
        return self.params[b:b + rows]

    def weight_grad(self, i):
        w, rows, kp, _ = self.layout[i]
        return self.grads[w:w + rows * kp].view(rows, kp)

    def bias_grad(self, i):
        _, rows, _, b = self.layout[i]
        return self.grads[b:b + rows]

    def _st(self):
        return nat.stream_handle(self.dev)

    def _refresh_bf16(self):
        nat.check(nat.lib().nn_cast_bf16(nat.ptr(self.params), 1, self.nparams, self.nparams,
                                         nat.ptr(self.params_bf16), self.nparams, None, 0, self._st()),
                  "nn cast")

    def _buffers(self, nb: int):
        """Workspace for the largest batch seen, and outputs: those of a batch
        of another size than the last are tensors of their own."""
        if nb > self._cap:
            nbytes = nat.lib().nn_net_workspace_bytes(self._table, len(self.layers), nb, 1)
            if nbytes < 0:
                raise ValueError(f"the network's shapes are not supported for a batch of {nb}")
            self._ws = torch.empty(int(nbytes), dtype=torch.uint8, device=self.dev)
            self._cap = nb
        if nb != self._nb:
            self.out = torch.empty((nb, self.controls), device=self.dev)
            self.dpred = torch.empty_like(self.out)
            self.loss = torch.zeros(1, device=self.dev)
            self._nb = nb

    # ----------------------------------------------------------- forward
    def forward(self, x: torch.Tensor) -> torch.Tensor:
        """x: gauge eta [Nb, gauges, samples] fp32 (metres) -> normalised
        controls [Nb, controls] fp32 (an internal buffer that the next call
        with as many records overwrites)."""
        x = nat.require_cuda_f32("x", x)
        nb, G, T = x.shape
        if G != self.gauges or T != self.samples:
            raise ValueError(f"expected [N, {self.gauges}, {self.samples}] gauge series, got {tuple(x.shape)}")
        self._buffers(nb)
        rc = nat.lib().nn_net_forward(self._table, len(self.layers), nat.ptr(self.params),
                                      nat.ptr(self.params_bf16), nat.ptr(x), INPUT_SCALE, nb,
                                      nat.ptr(self._ws), nat.ptr(self.out), self.wait_ns,
                                      nat.ptr(self.err), self._st())
        nat.check(rc, "nn forward")
        return self.out

    # ---------------------------------------------------------- backward
    def backward(self, dout: torch.Tensor) -> None:
        """Gradients of all parameters into self.grads for the cotangent of
        the last forward's output [Nb, controls]."""
        dout = nat.require_cuda_f32("dout", dout)
        rc = nat.lib().nn_net_backward(self._table, len(self.layers), nat.ptr(self.params_bf16),
                                       nat.ptr(dout), self._nb, nat.ptr(self._ws), nat.ptr(self.grads),
                                       self.wait_ns, nat.ptr(self.err), self._st())
        nat.check(rc, "nn backward")

    # ---------------------------------------------------------- training
    def loss_and_grad(self, x, y_norm) -> torch.Tensor:
        pred = self.forward(x)
        nb = pred.shape[0]
        rc = nat.lib().nn_mse(nat.ptr(pred), nat.ptr(y_norm), nb, self.controls, nat.ptr(self.loss),
                              nat.ptr(self.dpred), self._st())
        nat.check(rc, "nn mse")
        self.backward(self.dpred)
        return self.loss

    def adam_step(self, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8):
        self.step_count += 1
        rc = nat.lib().nn_adam_bf16(nat.ptr(self.params), nat.ptr(self.grads), nat.ptr(self.m),
                                    nat.ptr(self.v), self.nparams, lr, beta1, beta2, eps,
                                    self.step_count, nat.ptr(self.params_bf16), self._st())
        nat.check(rc, "nn adam")

    def train_step(self, x, y_norm, lr=1e-3):
        loss = self.loss_and_grad(x, y_norm)
        self.adam_step(lr)
        return loss

    def check_errors(self):
        code = int(self.err.item())
        if code & 2:
            raise RuntimeError(f"nn_gemm_bf16: tensor-core work had not finished when its tensor "
                               f"memory was freed (code {code:#x}); the CUDA context is suspect")
        if code != 0:
            raise RuntimeError(f"a bounded wait in nn_gemm_bf16 ran past its time limit (code {code:#x})")

    def predict_controls(self, gauges_eta: torch.Tensor, batch: int = 256) -> torch.Tensor:
        """Spline control values [N, controls] (metres) for gauge series
        [N, gauges, samples]."""
        outs = []
        for s in range(0, gauges_eta.shape[0], batch):
            y = self.forward(gauges_eta[s:s + batch].contiguous())
            outs.append(y * CONTROL_SCALE + CONTROL_MEAN)
        return torch.cat(outs)

    def state_dict(self):
        return {"params": self.params.detach().cpu(), "step": self.step_count}

    def load_state_dict(self, sd):
        self.params.copy_(sd["params"].to(self.dev))
        self.step_count = int(sd.get("step", 0))
        self._refresh_bf16()


def normalise_controls(values: torch.Tensor) -> torch.Tensor:
    return (values - CONTROL_MEAN) / CONTROL_SCALE


__all__ = ["WarmStartNet", "architecture", "param_layout", "normalise_controls", "Conv", "Dense",
           "SAMPLES", "GAUGES", "CONTROLS", "INPUT_SCALE", "CONTROL_MEAN", "CONTROL_SCALE"]
