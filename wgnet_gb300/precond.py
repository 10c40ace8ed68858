"""Learned update network for refinement (no reference counterpart: WGNet's refine(),
python/wgnet/refine.py:41-169, is plain projected L-BFGS).

`UpdateNet` maps (current 70x70 velocity in km/s, the exact misfit gradient, the band index) to a
proposed model update in km/s. It is a dilated residual convolution network, ~0.45 M parameters:

    features (8 channels: v - 3, g / rms(g), one-hot band x 4, depth, 0)
    conv3x3 8 -> 64, ReLU
    6 residual blocks, dilations 1, 2, 4, 8, 4, 2:  h = h + conv3x3_d1(ReLU(conv3x3_d(h)))
    conv3x3 64 -> 1 (x 0.25 km/s)

Weights are BF16 with FP32 master copies; every convolution, its data gradient and its weight gradient
run on the tensor cores with FP32 accumulation (`wg_pc_conv`, `wg_pc_conv_wgrad`), which read the
activations' shifted pixels directly and finish ReLU, residual adds, masks and bf16 casts in their
epilogues; only the 8-channel input goes through im2col columns. Features, loss and Adam are the
library's own kernels too. PyTorch only holds the buffers.
"""

from __future__ import annotations

import ctypes
import math
from dataclasses import dataclass

import numpy as np

from . import _lib
from ._lib import check

CIN = 8
CH = 64
DILATIONS = (1, 2, 4, 8, 4, 2)
OUT_SCALE = 0.25
BANDS = (6.0, 9.0, 12.0, None)
# epilogues of wg_pc_conv
FWD_RELU, FWD_FIRST, FWD_RESIDUAL, FWD_OUT, DGRAD_MASK, DGRAD_ADD, DGRAD_ADD_MASK = range(7)


def band_index(band_hz) -> int:
    return BANDS.index(band_hz) if band_hz in BANDS else 3


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    import torch

    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


@dataclass
class Layer:
    name: str
    cin: int
    n: int      # GEMM N (output channels, padded to 64)
    kp: int     # GEMM K (9 cin padded to 64)
    dil: int
    w32: object
    m1: object
    m2: object
    w: object   # bf16 [n][kp]
    wt: object  # bf16 [kp][n]


class UpdateNet:
    def __init__(self, seed: int = 0, device=None):
        import torch

        self._lib = _lib.load()
        self.device = torch.device(device or "cuda")
        g = np.random.default_rng(seed)
        self.layers: list[Layer] = []
        self._add("in", CIN, CH, 1, g, std=math.sqrt(2.0 / (9 * CIN)))
        for i, d in enumerate(DILATIONS):
            self._add(f"b{i}a", CH, CH, d, g, std=math.sqrt(2.0 / (9 * CH)))
            self._add(f"b{i}b", CH, CH, 1, g, std=0.1 * math.sqrt(2.0 / (9 * CH)))
        self._add("out", CH, CH, 1, g, std=1e-3, out_channels=1)
        self.step = 0
        self._bufs = {}
        self._status = torch.zeros(4, device=self.device, dtype=torch.int32)
        self._sync_bf16()

    # -- parameters ----------------------------------------------------------------------------
    def _add(self, name, cin, n, dil, g, std, out_channels=None):
        import torch

        k = 9 * cin
        kp = -(-k // 64) * 64
        w = np.zeros((n, kp), np.float32)
        rows = out_channels or n
        w[:rows, :k] = g.normal(0.0, std, (rows, k)).astype(np.float32)
        dev = self.device
        t = torch.from_numpy(w).to(dev)
        self.layers.append(Layer(name, cin, n, kp, dil, t, torch.zeros_like(t), torch.zeros_like(t),
                                 torch.empty((n, kp), device=dev, dtype=torch.bfloat16),
                                 torch.empty((kp, n), device=dev, dtype=torch.bfloat16)))

    def _adam(self, parts=None, grads=None, lr: float = 0.0):
        """One Adam step of every layer from its gradient partials (which also leaves the summed gradients
        in `grads`), or, without partials, a refresh of the bf16 weights."""
        n = len(self.layers)

        def array(kind, values):
            return (kind * n)(*values)

        def ptrs(tensors):
            return array(ctypes.c_void_p, [t.data_ptr() for t in tensors])

        Ls = self.layers
        check(self._lib.wg_pc_adam_layers(
            n, ptrs([parts[L.name] for L in Ls]) if parts else None,
            array(ctypes.c_int, [parts[L.name].shape[0] for L in Ls]) if parts else None,
            array(ctypes.c_int, [L.n for L in Ls]), array(ctypes.c_int, [L.kp for L in Ls]), ptrs([L.w32 for L in Ls]),
            ptrs([L.m1 for L in Ls]), ptrs([L.m2 for L in Ls]), ptrs([grads[L.name] for L in Ls]) if grads else None,
            ptrs([L.w for L in Ls]), ptrs([L.wt for L in Ls]), float(lr), 0.9, 0.999, 1e-8, self.step, _stream()), "adam")

    def _by_layer(self, flat) -> dict:
        sizes = [L.n * L.kp for L in self.layers]
        return {L.name: t.view(L.n, L.kp) for L, t in zip(self.layers, flat.split(sizes))}

    def _sync_bf16(self):
        self._adam()

    @property
    def parameters(self) -> int:
        total = 0
        for L in self.layers:
            rows = 1 if L.name == "out" else L.n
            total += rows * 9 * L.cin
        return total

    def state_dict(self) -> dict:
        return {L.name: L.w32.cpu().numpy() for L in self.layers} | {"step": np.array(self.step)}

    def load_state_dict(self, d: dict) -> None:
        import torch

        for L in self.layers:
            L.w32.copy_(torch.from_numpy(np.asarray(d[L.name], np.float32)))
            L.m1.zero_()
            L.m2.zero_()
        self.step = int(d.get("step", 0))
        self._sync_bf16()

    def save(self, path) -> None:
        np.savez(path, **self.state_dict())

    @classmethod
    def load(cls, path, device=None) -> "UpdateNet":
        net = cls(device=device)
        with np.load(path) as d:
            net.load_state_dict({k: d[k] for k in d.files})
        return net

    # -- building blocks ------------------------------------------------------------------------
    def _buf(self, key, shape, dtype):
        import torch

        b = self._bufs.get(key)
        if b is None or tuple(b.shape) != tuple(shape) or b.dtype != dtype:
            b = torch.empty(shape, device=self.device, dtype=dtype)
            self._bufs[key] = b
        return b

    def _conv(self, mode, L: Layer, x, shape, out16=None, out32=None, add=None, mask=None):
        """One fused convolution (modes of wg_pc_conv); the data-gradient modes take L's transposed
        weights."""
        B, H, W = shape
        ptr = lambda t: None if t is None else _p(t)  # noqa: E731
        check(self._lib.wg_pc_conv(mode, _p(x), B, H, W, L.dil, _p(L.wt if mode >= DGRAD_MASK else L.w), L.kp, ptr(add),
                                   ptr(mask), ptr(out32), ptr(out16), _p(self._status), _stream()), "conv")

    def _wgrad(self, L: Layer, x, dy16, shape, splits, columns=0):
        """Weight gradient partials of L from its input (or the input's columns) and the bf16 dL/dy."""
        import torch

        B, H, W = shape
        nz = self._lib.wg_pc_wgrad_partials(B, H, W, splits)
        part = torch.empty((max(nz, 1), L.kp, L.n), device=self.device, dtype=torch.float32)
        check(self._lib.wg_pc_conv_wgrad(_p(x), columns, _p(dy16), B, H, W, L.dil, splits, _p(part), _p(self._status),
                                         _stream()), "gemm wgrad")
        return part

    # -- forward / training -----------------------------------------------------------------------
    def forward(self, vel_km, grad, band, keep: bool = False):
        """`vel_km`, `grad`: [B, H, W] float32 CUDA tensors; `band`: [B] int32 CUDA tensor of band
        indices (0..3 for 6, 9, 12 Hz and the full band). Returns the proposed update [B, H, W]
        (km/s)."""
        import torch

        if not hasattr(self, "_bufs"):
            self._bufs = {}
            self._status = torch.zeros(4, device=self.device, dtype=torch.int32)
        B, H, W = vel_km.shape
        M = B * H * W
        shape = (B, H, W)

        def bf16(cols):
            return torch.empty((M, cols), device=self.device, dtype=torch.bfloat16)

        def f32():
            return torch.empty((M, CH), device=self.device, dtype=torch.float32)

        rms = self._buf("rms", (B,), torch.float32)
        x0 = bf16(CIN)
        check(self._lib.wg_pc_features(_p(vel_km.contiguous()), _p(grad.contiguous()), _p(band.contiguous()), B, H,
                                       W, _p(rms), _p(x0), _stream()), "features")
        L = self.layers[0]
        col = bf16(L.kp)
        check(self._lib.wg_pc_im2col(_p(x0), B, H, W, L.cin, L.dil, L.kp, _p(col), _stream()), "im2col")
        h16, h = bf16(CH), f32()
        self._conv(FWD_FIRST, L, col, shape, out16=h16, out32=h)
        saved = {"x0": x0, "shape": shape, "h0": h16, "col0": col}
        blocks = []
        a16 = None
        for i in range(len(DILATIONS)):
            La, Lb = self.layers[1 + 2 * i], self.layers[2 + 2 * i]
            if a16 is None or keep:
                a16 = bf16(CH)
            self._conv(FWD_RELU, La, h16, shape, out16=a16)
            # the block's output; without `keep` it takes its input's place (the second convolution
            # reads a16 only)
            hn, hn16 = (f32(), bf16(CH)) if keep else (h, h16)
            self._conv(FWD_RESIDUAL, Lb, a16, shape, out16=hn16, out32=hn, add=h)
            blocks.append((h16, a16, h))
            h, h16 = hn, hn16
        out = torch.empty(M, device=self.device, dtype=torch.float32)
        self._conv(FWD_OUT, self.layers[-1], h16, shape, out32=out)
        if keep:
            saved["blocks"] = blocks
            saved["hlast"] = h16
            saved["hlast32"] = h
            self._saved = saved
            self._out = out
            self.last_activations = saved
        return (out * OUT_SCALE).view(B, H, W)

    def train_step(self, vel_km, grad, band, target_km, lr: float = 1e-3, splits: int = 64) -> float:
        """One Adam step on the mean squared error between the proposed update and `target_km`
        ([B, H, W], km/s). B must be a multiple of 16 (the weight-gradient reduction runs over
        B H W rows in tiles of 64). Returns the loss."""
        import torch

        self.forward(vel_km, grad, band, keep=True)
        s = self._saved
        shape = s["shape"]
        B, H, W = shape
        M = B * H * W
        dout = torch.empty(M, device=self.device, dtype=torch.float32)
        loss = torch.zeros(1, device=self.device, dtype=torch.float64)
        check(self._lib.wg_pc_mse(_p(self._out), 1, _p(target_km.contiguous()), OUT_SCALE, M, _p(loss), _p(dout),
                                  _stream()), "mse")
        parts = {}
        Lo = self.layers[-1]
        dh = torch.empty((M, CH), device=self.device, dtype=torch.float32)
        dh16 = torch.empty((M, CH), device=self.device, dtype=torch.bfloat16)
        dout16 = torch.empty((M, CH), device=self.device, dtype=torch.bfloat16)
        check(self._lib.wg_pc_out_dgrad(_p(dout), _p(Lo.wt), B, H, W, _p(dh), _p(dh16), _p(dout16), _stream()), "out dgrad")
        parts["out"] = self._wgrad(Lo, s["hlast"], dout16, shape, splits)
        t16 = dout16  # read for the last time above
        for i in reversed(range(len(DILATIONS))):
            La, Lb = self.layers[1 + 2 * i], self.layers[2 + 2 * i]
            h16, a16, _ = s["blocks"][i]
            parts[Lb.name] = self._wgrad(Lb, a16, dh16, shape, splits)
            self._conv(DGRAD_MASK, Lb, dh16, shape, out16=t16, mask=a16)
            parts[La.name] = self._wgrad(La, h16, t16, shape, splits)
            if i:
                self._conv(DGRAD_ADD, La, t16, shape, out16=dh16, out32=dh, add=dh)
            else:
                self._conv(DGRAD_ADD_MASK, La, t16, shape, out16=dh16, add=dh, mask=s["h0"])
        Li = self.layers[0]
        parts["in"] = self._wgrad(Li, s["col0"], dh16, shape, splits, columns=Li.kp)
        self.step += 1
        flat = torch.empty(sum(L.n * L.kp for L in self.layers), device=self.device, dtype=torch.float32)
        self._adam(parts, self._by_layer(flat), lr)
        self._last_grads = flat
        self._saved = None
        self.last_activations = None
        return float(loss.item())

    def status(self) -> int:
        """Device status word of the GEMM pipeline (non-zero after a timed-out wait)."""
        return int(self._status[0].item())

    def weight_gradients(self) -> dict:
        """{layer: dL/dW [n][kp]} of the last train_step (for tests)."""
        return self._by_layer(self._last_grads.clone())


__all__ = ["UpdateNet", "BANDS", "band_index", "DILATIONS", "OUT_SCALE"]
