"""BRF surrogate: an MLP from (r_eff, lambda, cos theta0, depth) to the 648-bin BRF and albedo.

The reference's only route to a BRF is the Monte Carlo walk followed by the
histogram arithmetic of post_processing.py:46-100.  This module learns that map
from walks the GPU walk itself produces, so a BRF can be predicted in
microseconds; plain Monte Carlo stays the fallback outside the training hull or
where the ensemble disagrees, and the judge of the network's error.

Network: 4 -> 256 -> 256 -> 256 -> 649, SiLU, BF16 weights and activations on
tensor cores with FP32 accumulation (include/mcw_mlp.h: inference is one fused
tcgen05 kernel with tensor-memory accumulators whose hidden activations never leave
shared memory; training runs layer-by-layer GEMMs that keep the pre-activations for
the backward pass), FP32 master weights and Adam.  ``MLPFunction`` is the torch.autograd.Function whose forward and backward
run those kernels; inputs and outputs are torch CUDA tensors, PyTorch is only the
container.  Targets are standardised log(BRF / albedo + 0.02) per bin and
log(albedo).
"""
import ctypes
import math
from dataclasses import dataclass

import numpy as np

from . import _abi

DIMS = (4, 256, 256, 256, 649)
N_BRF = 648
BRF_FLOOR = 0.02
# training hull: the parameter ranges the surrogate is trained and judged on
R_RANGE = (50.0, 1500.0)      # r_eff [um], log-uniform
WVL_RANGE = (0.9, 1.8)        # centre wavelength [um]
MU_RANGE = (0.3, 1.0)         # cos theta0
DEPTH_RANGE = (0.01, 1.0)     # [m], log-uniform


def encode(r_eff, wvl, mu0, depth):
    """Inputs scaled to [-1, 1] over the training hull, float32 [n, 4]."""
    r = np.log(np.asarray(r_eff, np.float64))
    d = np.log(np.asarray(depth, np.float64))
    x = np.stack([
        2 * (r - math.log(R_RANGE[0])) / (math.log(R_RANGE[1]) - math.log(R_RANGE[0])) - 1,
        2 * (np.asarray(wvl, np.float64) - WVL_RANGE[0]) / (WVL_RANGE[1] - WVL_RANGE[0]) - 1,
        2 * (np.asarray(mu0, np.float64) - MU_RANGE[0]) / (MU_RANGE[1] - MU_RANGE[0]) - 1,
        2 * (d - math.log(DEPTH_RANGE[0])) / (math.log(DEPTH_RANGE[1]) - math.log(DEPTH_RANGE[0])) - 1,
    ], axis=-1)
    return x.astype(np.float32)


def hull():
    """Origin and width of log r_eff, wavelength, mu0 and log depth, as encode scales them."""
    out = []
    for lo, hi in ((math.log(R_RANGE[0]), math.log(R_RANGE[1])), WVL_RANGE, MU_RANGE,
                   (math.log(DEPTH_RANGE[0]), math.log(DEPTH_RANGE[1]))):
        out += [lo, hi - lo]
    return out


def in_hull(r_eff, wvl, mu0, depth):
    x = encode(r_eff, wvl, mu0, depth)
    return np.all(np.abs(x) <= 1.0 + 1e-6, axis=-1)


def to_target(brf, albedo):
    """Network target space: log(BRF / albedo + floor) per bin (the shape, about 1 on
    average) and log(albedo), so every bin keeps relative precision."""
    a = np.maximum(np.asarray(albedo, np.float64), 1e-6)
    shape = np.maximum(np.asarray(brf, np.float64), 0) / a[:, None]
    return np.concatenate([np.log(shape + BRF_FLOOR), np.log(a)[:, None]], axis=1).astype(np.float32)


def from_target(y):
    y = np.asarray(y, np.float64)
    a = np.exp(y[:, N_BRF])
    return (np.exp(y[:, :N_BRF]) - BRF_FLOOR) * a[:, None], a


# ------------------------------------------------------------------ kernels

def _stream(torch):
    """The current stream's handle (a plain integer; making the Stream object takes several us)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def _ptr(t):
    return t.data_ptr() if t is not None else None


def _gemm(torch, epi, m, n, k, a, lda, b, ldb, c, ldc, trans_a=0, trans_b=0, bias=None, aux=None,
          ldaux=0, c2=None, ldc2=0, engine=_abi.ENGINE_MMA_SYNC):
    g = _abi.GemmC(m, n, k, trans_a, trans_b, epi, a.data_ptr(), lda, ldb, b.data_ptr(),
                   bias.data_ptr() if bias is not None else None,
                   aux.data_ptr() if aux is not None else None, ldaux, ldc, c.data_ptr(),
                   c2.data_ptr() if c2 is not None else None, ldc2, engine)
    rc = _abi.load().mcw_mlp_gemm(ctypes.byref(g), _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_gemm failed (m=%d n=%d k=%d)' % (m, n, k))


def _cast(torch, x):
    y = torch.empty(x.shape, dtype=torch.bfloat16, device=x.device)
    rc = _abi.load().mcw_mlp_cast_bf16(_ptr(x), _ptr(y), x.numel(), _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_cast_bf16 failed')
    return y


# engine of training's GEMMs (forward with kept pre-activations, and the backward
# layouts: transposed operands, silu' epilogue); inference runs the fused tcgen05
# kernel (forward_fused)
TRAIN_ENGINE = _abi.ENGINE_TCGEN05


def pack_weights(torch, w16):
    """All four weight matrices in the tensor-core operand layout of mcw_mlp_forward."""
    blob = torch.empty(_abi.MLP_PACK_BYTES, dtype=torch.uint8, device=w16[0].device)
    rc = _abi.load().mcw_mlp_pack(_ptr(w16[0]), _ptr(w16[1]), _ptr(w16[2]), _ptr(w16[3]), _ptr(blob),
                                  _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_pack failed')
    return blob


# row pitch of the fused kernel's output: 649 values rounded up to 16 bytes (its
# 16-byte stores): 652 floats or 656 halves
Y_PITCH = 652
Y_PITCH_F16 = 656


def forward_fused(torch, x, w16, biases, blob, half=False):
    """Inference of the whole network in one kernel (mcw_mlp_forward, or
    mcw_mlp_forward_f16 with half=True: outputs rounded to fp16, half the bytes);
    x float32 [m, 4]; returns a [m, 649] view of the output rows."""
    if x.dtype != torch.float32 or not x.is_contiguous():
        x = x.contiguous().float()
    m = x.shape[0]
    pitch = Y_PITCH_F16 if half else Y_PITCH
    y = torch.empty((m, pitch), dtype=torch.float16 if half else torch.float32, device=x.device)
    b1, b2, b3, b4 = [t if t.is_contiguous() else t.contiguous() for t in biases]
    L = _abi.load()
    fn = L.mcw_mlp_forward_f16 if half else L.mcw_mlp_forward
    rc = fn(x.data_ptr(), m, b1.data_ptr(), b2.data_ptr(), b3.data_ptr(), b4.data_ptr(), blob.data_ptr(), y.data_ptr(),
            pitch, _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_forward failed (m=%d)' % m)
    return y[:, :DIMS[-1]]


def forward_ensemble(torch, x, blob, bias, members):
    """Inference of an ensemble's members on the same inputs in one launch
    (mcw_mlp_forward_ensemble_f16): blob holds the members' packed weights one after the
    other (members x MLP_PACK_BYTES), bias their biases (float32 [members, 1417], b1 | b2 |
    b3 | b4); returns fp16 [members, m, 649] views of the output rows, each member's equal
    to forward_fused(half=True) of that member."""
    x = x.contiguous().float()
    m = x.shape[0]
    y = torch.empty((members, m, Y_PITCH_F16), dtype=torch.float16, device=x.device)
    rc = _abi.load().mcw_mlp_forward_ensemble_f16(_ptr(x), m, members, _ptr(bias), _ptr(blob), _ptr(y),
                                                  Y_PITCH_F16, _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_forward_ensemble_f16 failed (m=%d, members=%d)' % (m, members))
    return y[:, :, :DIMS[-1]]


def _cast_rows(torch, t, colsum=None):
    """t [m, n] (f32 or bf16) as bf16 rows of a whole number of 16 bytes, zero past n (what the
    TMA-fed products read): [m, n rounded up to 8].  colsum: [ceil(m / 128), n] f32 for the column
    sums of t over every 128 rows."""
    t = t.contiguous()
    m, n = t.shape
    out = torch.empty((m, _align8(n)), dtype=torch.bfloat16, device=t.device)
    rc = _abi.load().mcw_mlp_cast_rows(_ptr(t), int(t.dtype == torch.bfloat16), m, n, n, _ptr(out), out.shape[1],
                                       _ptr(colsum), n, _stream(torch))
    if rc:
        raise _abi.McwError(rc, 'mcw_mlp_cast_rows failed')
    return out


def _rows16(torch, t):
    """t (bf16) itself when its rows are whole 16-byte runs, else padded."""
    return t if t.shape[1] % 8 == 0 and t.is_contiguous() and t.data_ptr() % 16 == 0 else _cast_rows(torch, t)


def forward_cached(torch, x16, w16, biases, keep=True):
    """Forward pass on the tensor-core kernels; returns (y fp32, cache for backward).
    keep=False (inference) skips storing the FP32 pre-activations."""
    m = x16.shape[0]
    a = _rows16(torch, x16)
    zs, acts = [], [a]
    for layer in range(3):
        n, k = w16[layer].shape
        w = _rows16(torch, w16[layer])
        z = torch.empty((m, n), dtype=torch.float32, device=x16.device) if keep else None
        nxt = torch.empty((m, n), dtype=torch.bfloat16, device=x16.device)
        _gemm(torch, _abi.EPI_BIAS_SILU, m, n, min(k, DIMS[layer]), a, a.shape[1], w, w.shape[1], nxt, n,
              bias=biases[layer], c2=z, ldc2=n, engine=TRAIN_ENGINE)
        zs.append(z)
        acts.append(nxt)
        a = nxt
    n, k = w16[3].shape
    y = torch.empty((m, n), dtype=torch.float32, device=x16.device)
    _gemm(torch, _abi.EPI_BIAS_F32, m, n, k, a, k, w16[3], k, y, n, bias=biases[3], engine=TRAIN_ENGINE)
    return y, (zs, acts)


def backward_cached(torch, gy, w16, cache, need_dx=True):
    """Backward pass: gradients of the weights, biases and (optionally) the input.  Three products
    down the layers, whose epilogues leave the column sums of every 128 rows, then the four weight
    gradients in one launch, which also adds up the bias gradients: the operands are read where
    they lie, transposed by the tensor core."""
    zs, acts = cache[0], [_rows16(torch, a) for a in cache[1]]
    m = gy.shape[0]
    dev = gy.device
    blocks = (m + 127) // 128
    f32 = torch.float32
    sums = [torch.empty((blocks, w.shape[0]), dtype=f32, device=dev) for w in w16]
    g16 = [None] * 3 + [_cast_rows(torch, gy.float(), colsum=sums[3])]
    st = _stream(torch)
    L = _abi.load()
    for layer in (3, 2, 1):
        # G_prev[b, i] = (sum_o G[b, o] W[o, i]) * silu'(Z_prev[b, i])
        n_out, k_in = w16[layer].shape
        g, w = g16[layer], _rows16(torch, w16[layer])
        prev = torch.empty((m, k_in), dtype=torch.bfloat16, device=dev)
        q = _abi.GemmProblemC(m=m, n=k_in, k=n_out, groups=1, splits=1, epilogue=_abi.EPI_DSILU, a=g.data_ptr(),
                              lda=g.shape[1], b=w.data_ptr(), ldb=w.shape[1], trans_b=1,
                              aux=zs[layer - 1].data_ptr(), ldaux=k_in, c=prev.data_ptr(), ldc=k_in,
                              colsum=sums[layer - 1].data_ptr(), ld_colsum=k_in)
        rc = L.mcw_mlp_gemm_batch(ctypes.byref(q), 1, st)
        if rc:
            raise _abi.McwError(rc, 'backward product failed (layer %d)' % layer)
        g16[layer - 1] = prev
    dx = None
    if need_dx:
        n_out, k_in = w16[0].shape
        w = _rows16(torch, w16[0])
        dx = torch.empty((m, DIMS[0]), dtype=f32, device=dev)
        _gemm(torch, _abi.EPI_F32, m, DIMS[0], n_out, g16[0], n_out, w, w.shape[1], dx, DIMS[0], trans_b=1,
              engine=TRAIN_ENGINE)
    # dW[o, i] = sum_b G[b, o] A[b, i], db[o] = sum_b G[b, o]
    dws = [torch.empty((w.shape[0], DIMS[layer]), dtype=f32, device=dev) for layer, w in enumerate(w16)]
    dbs = [torch.empty(w.shape[0], dtype=f32, device=dev) for w in w16]
    calls = (_abi.GemmProblemC * 4)()
    for layer, w in enumerate(w16):
        n_out, k_in = dws[layer].shape
        calls[layer] = _abi.GemmProblemC(
            m=n_out, n=k_in, k=m, groups=1, splits=1, epilogue=_abi.EPI_F32, a=g16[layer].data_ptr(),
            lda=g16[layer].shape[1], b=acts[layer].data_ptr(), ldb=acts[layer].shape[1], trans_a=1, trans_b=1,
            c=dws[layer].data_ptr(), ldc=k_in, colsum=dbs[layer].data_ptr(), colsum_in=sums[layer].data_ptr(),
            ld_colsum=n_out, colsum_chunks=blocks)
    rc = L.mcw_mlp_gemm_batch(calls, 4, st)
    if rc:
        raise _abi.McwError(rc, 'weight gradients failed (m=%d)' % m)
    return dx, dws, dbs


def forward_tangent(torch, x16, xdot16, w16, biases):
    """Network outputs and their directional derivative along the input tangent xdot,
    in one forward pass on the tensor-core kernels (forward mode: 4 more GEMMs, not one
    backward pass per output).  x16, xdot16 bf16 [n, 4]; returns (y, ydot) fp32 [n, 649].
    Per layer: hdot_l = (hdot_{l-1} W_l^T) * silu'(z_l), the SiLU' epilogue of the backward
    GEMMs with the pre-activations z_l of the forward pass; ydot = hdot_3 W_4^T."""
    w16 = [_rows16(torch, w) for w in w16]
    y, (zs, _) = forward_cached(torch, x16, w16, biases, keep=True)
    m = x16.shape[0]
    t = _rows16(torch, xdot16)
    for layer in range(3):
        n, k = w16[layer].shape
        nxt = torch.empty((m, n), dtype=torch.bfloat16, device=x16.device)
        _gemm(torch, _abi.EPI_DSILU, m, n, min(k, DIMS[layer]), t, t.shape[1], w16[layer], k, nxt, n, aux=zs[layer],
              ldaux=n, engine=TRAIN_ENGINE)
        t = nxt
    n, k = w16[3].shape
    ydot = torch.empty((m, n), dtype=torch.float32, device=x16.device)
    _gemm(torch, _abi.EPI_F32, m, n, k, t, k, w16[3], k, ydot, n, engine=TRAIN_ENGINE)
    return y, ydot


class EnsembleTangent:
    """forward_tangent of every member of an ensemble on the same n inputs, each product one launch
    for all members: the members' bf16 weights laid side by side and the buffers of one batch size,
    made once for the evaluations of a retrieval.  The tangent is that of the first input, dx0."""

    def __init__(self, torch, members, n, dx0):
        self.torch = torch
        self.n, self.G = n, len(members)
        G, H, N, dev = self.G, DIMS[1], DIMS[-1], members[0].w16[0].device
        bf16, f32 = torch.bfloat16, torch.float32
        ws = [torch.stack([_rows16(torch, m.w16[layer]) for m in members]) for layer in range(4)]
        bs = [torch.stack([m.params[2 * layer + 1].float() for m in members]) for layer in range(4)]
        self.x = torch.zeros((G, n, 8), dtype=bf16, device=dev)
        xdot = torch.zeros((G, n, 8), dtype=bf16, device=dev)
        xdot[:, :, 0] = dx0
        h = [torch.empty((G, n, H), dtype=bf16, device=dev) for _ in range(3)]
        t = [torch.empty((G, n, H), dtype=bf16, device=dev) for _ in range(3)]
        z = [torch.empty((G, n, H), dtype=f32, device=dev) for _ in range(3)]
        self.y = torch.empty((G, n, Y_PITCH), dtype=f32, device=dev)
        self.ydot = torch.empty((G, n, Y_PITCH), dtype=f32, device=dev)
        self.keep = (ws, bs, xdot, h, t, z)

        def call(epi, layer, a, c, **more):
            w = ws[layer]
            return _abi.GemmProblemC(m=n, n=w.shape[1], k=DIMS[layer], groups=G, splits=1, epilogue=epi, a=a.data_ptr(),
                                     lda=a.shape[2], stride_a=n * a.shape[2], b=w.data_ptr(), ldb=w.shape[2],
                                     stride_b=w.shape[1] * w.shape[2], c=c.data_ptr(), ldc=c.shape[2],
                                     stride_c=n * c.shape[2], **more)
        self.calls = []
        a, d = self.x, xdot
        for layer in range(3):
            zl = dict(c2=z[layer].data_ptr(), ldc2=H, stride_c2=n * H)
            self.calls.append(call(_abi.EPI_BIAS_SILU, layer, a, h[layer], bias=bs[layer].data_ptr(), stride_bias=H, **zl))
            self.calls.append(call(_abi.EPI_DSILU, layer, d, t[layer], aux=z[layer].data_ptr(), ldaux=H, stride_aux=n * H))
            a, d = h[layer], t[layer]
        self.calls.append(call(_abi.EPI_BIAS_F32, 3, a, self.y, bias=bs[3].data_ptr(), stride_bias=N))
        self.calls.append(call(_abi.EPI_F32, 3, d, self.ydot))

    def run(self, x):
        """x float32 [n, 4], or None for what self.x (bf16 [members, n, 8]) holds; returns (y, ydot)
        fp32 [members, n, Y_PITCH], 649 columns used; valid until the next call."""
        if x is not None:
            self.x[:, :, :DIMS[0]] = x
        L, st = _abi.load(), _stream(self.torch)
        for c in self.calls:
            rc = L.mcw_mlp_gemm_batch(ctypes.byref(c), 1, st)
            if rc:
                raise _abi.McwError(rc, 'ensemble tangent failed (n=%d)' % self.n)
        return self.y, self.ydot


def _mlp_function():
    import torch

    class MLPFunction(torch.autograd.Function):
        """y = MLP(x) on the BF16 tensor-core kernels; params are FP32 masters
        (W1, b1, ..., W4, b4).  Backward returns FP32 gradients for x and every
        parameter."""

        @staticmethod
        def forward(ctx, x, *params):
            ws, bs = params[0::2], params[1::2]
            w16 = [_cast(torch, w.contiguous()) for w in ws]
            x16 = _cast(torch, x.contiguous().float())
            y, cache = forward_cached(torch, x16, w16, [b.contiguous() for b in bs])
            ctx.save_for_backward(*w16, *cache[0], *cache[1])
            return y

        @staticmethod
        def backward(ctx, gy):
            saved = ctx.saved_tensors
            w16, zs, acts = list(saved[:4]), list(saved[4:7]), list(saved[7:11])
            dx, dws, dbs = backward_cached(torch, gy, w16, (zs, acts), need_dx=ctx.needs_input_grad[0])
            out = [dx]
            for dw, db in zip(dws, dbs):
                out += [dw, db]
            return tuple(out)

    return MLPFunction


_MLP_FN = None


def mlp_apply(x, params):
    global _MLP_FN
    if _MLP_FN is None:
        _MLP_FN = _mlp_function()
    return _MLP_FN.apply(x, *params)


# ------------------------------------------------------------------ model

class SurrogateMLP:
    """One network: FP32 master weights, BF16 copies, Adam moments (torch CUDA tensors)."""

    def __init__(self, seed=0, device='cuda'):
        import torch
        self.torch = torch
        g = torch.Generator(device='cpu').manual_seed(int(seed))
        self.params = []
        for fan_in, fan_out in zip(DIMS[:-1], DIMS[1:]):
            bound = math.sqrt(6.0 / fan_in) if fan_out != DIMS[-1] else math.sqrt(3.0 / fan_in)
            w = (torch.rand((fan_out, fan_in), generator=g) * 2 - 1) * bound
            self.params += [w.to(device), torch.zeros(fan_out, device=device)]
        self.m = [torch.zeros_like(p) for p in self.params]
        self.v = [torch.zeros_like(p) for p in self.params]
        self.w16 = [_cast(torch, w) for w in self.params[0::2]]
        self.step = 0
        self.y_mean = None
        self.y_std = None
        self._blob = None
        self._blob_key = None

    def packed(self):
        """Packed weights for the fused inference kernel, rebuilt when the weights change."""
        key = (self.step, tuple(w.data_ptr() for w in self.w16))
        if self._blob is None or self._blob_key != key:
            self._blob = pack_weights(self.torch, self.w16)
            self._blob_key = key
        return self._blob

    def predict_std(self, x, half=True):
        """Standardised outputs for encoded inputs x (torch CUDA float32 [n, 4]) from the
        fused inference kernel; fp16 by default (its rounding, 2^-11 relative, is below the
        network's bf16 activations), float32 with half=False."""
        return forward_fused(self.torch, x, self.w16, self.params[1::2], self.packed(), half=half)

    def train_step(self, x16, t, w_out, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8):
        """One Adam step on a batch (x16 bf16 [b, 4], t fp32 standardised targets)."""
        torch = self.torch
        m = x16.shape[0]
        y, cache = forward_cached(torch, x16, self.w16, self.params[1::2])
        n = y.shape[1]
        grad = torch.empty_like(y)
        grad16 = torch.empty((m, n), dtype=torch.bfloat16, device=y.device)
        loss = torch.zeros(1, dtype=torch.float32, device=y.device)
        L = _abi.load()
        rc = L.mcw_mlp_loss(_ptr(y), n, _ptr(t), n, _ptr(w_out), m, n, _ptr(grad), n, _ptr(grad16), n,
                            _ptr(loss), _stream(torch))
        if rc:
            raise _abi.McwError(rc, 'mcw_mlp_loss failed')
        _, dws, dbs = backward_cached(torch, grad, self.w16, cache, need_dx=False)
        self.step += 1
        grads = []
        for dw, db in zip(dws, dbs):
            grads += [dw, db]
        for i, (p, gr) in enumerate(zip(self.params, grads)):
            w16 = self.w16[i // 2] if i % 2 == 0 else None
            rc = L.mcw_mlp_adam(_ptr(p), _ptr(gr), _ptr(self.m[i]), _ptr(self.v[i]), _ptr(w16), p.numel(),
                                lr, beta1, beta2, eps, self.step, _stream(torch))
            if rc:
                raise _abi.McwError(rc, 'mcw_mlp_adam failed')
        return loss


# ------------------------------------------------------------------ training engine

IN_PAD = 16        # layer-1 inputs padded to 16: one 16-byte TMA row, one MMA K step


def _align8(n):
    return (n + 7) // 8 * 8


def flat_layout():
    """Layout of one member's parameters in the training engine's flat vectors.

    Returns (lay, P, tlay, T): lay['W%d'] = (offset, rows, cols) of W_l [out, in]
    (layer 1's inputs padded to IN_PAD columns, held at zero), lay['b%d'] = (offset, n);
    P elements per member; tlay['W%d'] = (offset, ld) of the transposed bf16 copy
    W_l^T [in, ld] (ld = out rounded up to 8) of W2, W3, W4 that Adam keeps beside the
    weights; T elements per member.  Every block starts on 8 elements."""
    lay, off = {}, 0
    for layer, (fan_in, fan_out) in enumerate(zip(DIMS[:-1], DIMS[1:])):
        k = IN_PAD if layer == 0 else fan_in
        lay['W%d' % layer] = (off, fan_out, k)
        off = _align8(off + fan_out * k)
        lay['b%d' % layer] = (off, fan_out)
        off = _align8(off + fan_out)
    tlay, toff = {}, 0
    for layer in (1, 2, 3):
        _, rows, cols = lay['W%d' % layer]
        ld = _align8(rows)
        tlay['W%d' % layer] = (toff, ld)
        toff += cols * ld
    return lay, off, tlay, toff


def _dw_splits(rows):
    """Split-K of the weight-gradient products over `rows` batch rows: about 1,024 rows
    per split, at most 64 splits, in the form mcw_mlp_gemm_grouped accepts."""
    chunks = (rows + 63) // 64
    want = max(1, min(64, rows // 1024))
    per = (chunks + want - 1) // want
    return (chunks + per - 1) // per


class EnsembleTrainer:
    """Adam steps of every member of an ensemble at once on the training engine
    (include/mcw_mlp.h): per step one gather of the members' batches, the three hidden
    products (bias + SiLU epilogues keeping pre-activations), the output product whose
    epilogue is the loss and its gradient, three products back down the layers, all
    weight and bias gradients, Adam over the flat parameters and the step counter, each
    one launch for all members.  Parameters live in flat [members, P] vectors
    (flat_layout).  The step is captured in a CUDA graph on first use and replayed;
    learning rate, step count and batch counter are device scalars, so the graph never
    changes."""

    def __init__(self, members, batch, x_all, t_all, w_out, lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8,
                 use_graph=True):
        import torch
        self.torch = torch
        self.members = members
        self.G = len(members)
        self.B = int(batch)
        self.beta1, self.beta2, self.eps = beta1, beta2, eps
        self.use_graph = use_graph
        self.graph = None
        G, B = self.G, self.B
        self.lay, self.P, self.tlay, self.T = flat_layout()
        dev = 'cuda'
        f32, bf16, i32 = torch.float32, torch.bfloat16, torch.int32
        # parameters, gradients, Adam moments and the bf16 copies (zeros in the padding)
        self.params = torch.zeros((G, self.P), dtype=f32, device=dev)
        self.m = torch.zeros_like(self.params)
        self.v = torch.zeros_like(self.params)
        self.grad = torch.zeros_like(self.params)
        for g, net in enumerate(members):
            for layer in range(4):
                o, rows, cols = self.lay['W%d' % layer]
                w = net.params[2 * layer]
                blk = self.params[g, o:o + rows * cols].view(rows, cols)
                blk[:, :w.shape[1]].copy_(w)
                ob, nb = self.lay['b%d' % layer]
                self.params[g, ob:ob + nb].copy_(net.params[2 * layer + 1])
                mw, vw = net.m[2 * layer], net.v[2 * layer]
                self.m[g, o:o + rows * cols].view(rows, cols)[:, :w.shape[1]].copy_(mw)
                self.v[g, o:o + rows * cols].view(rows, cols)[:, :w.shape[1]].copy_(vw)
                self.m[g, ob:ob + nb].copy_(net.m[2 * layer + 1])
                self.v[g, ob:ob + nb].copy_(net.v[2 * layer + 1])
        self.w16 = self.params.to(bf16)
        self.wt = torch.zeros((G, self.T), dtype=bf16, device=dev)
        for layer in (1, 2, 3):
            o, rows, cols = self.lay['W%d' % layer]
            to, ld = self.tlay['W%d' % layer]
            self.wt[:, to:to + cols * ld].view(G, cols, ld)[:, :, :rows].copy_(
                self.w16[:, o:o + rows * cols].view(G, rows, cols).transpose(1, 2))
        # data (inputs padded to IN_PAD, bf16) and the step's batch
        n_rows = x_all.shape[0]
        if n_rows < B:
            raise ValueError('fewer rows (%d) than the batch (%d)' % (n_rows, B))
        self.n_rows = n_rows
        self.x_all = torch.zeros((n_rows, IN_PAD), dtype=bf16, device=dev)
        self.x_all[:, :DIMS[0]].copy_(x_all.to(bf16))
        self.t_all = t_all.contiguous().float()
        self.w_out = w_out.contiguous().float()
        self.perm = torch.zeros((G, n_rows), dtype=i32, device=dev)
        self.counter = torch.zeros(1, dtype=i32, device=dev)
        self.step = torch.full((1,), max(int(net.step) for net in members) + 1, dtype=i32, device=dev)
        self.lr = torch.full((1,), float(lr), dtype=f32, device=dev)
        self.loss = torch.zeros(G, dtype=f32, device=dev)
        H, N = DIMS[1], DIMS[-1]
        self.x16 = torch.zeros((G, B, IN_PAD), dtype=bf16, device=dev)
        self.t = torch.zeros((G, B, N), dtype=f32, device=dev)
        self.h = [torch.zeros((G, B, H), dtype=bf16, device=dev) for _ in range(3)]
        self.z = [torch.zeros((G, B, H), dtype=f32, device=dev) for _ in range(3)]
        # gradients of the layers' outputs (the last with pitch 656)
        widths = [_align8(n) for n in (H, H, H, N)]
        self.g16 = [torch.zeros((G, B, n), dtype=bf16, device=dev) for n in widths]
        self.g32 = [torch.zeros((G, B, n), dtype=f32, device=dev) for n in widths]
        # bias gradients: rows summed in chunks of 1,024 when the batch is large, then in order
        self.colsum_rows = 1024 if B > 2048 else B
        self.splits = _dw_splits(B)
        if self.splits > 1:
            self.part = [torch.zeros((self.splits, G, rows * cols), dtype=f32, device=dev)
                         for (_, rows, cols) in (self.lay['W%d' % q] for q in range(4))]
        self._build_calls()

    # ---- the calls of one step, built once (pointers never change)
    def _gemm(self, epi, m, n, k, a, lda, sa, b, ldb, sb, c, ldc, sc, **more):
        return _abi.GemmProblemC(m=m, n=n, k=k, groups=self.G, splits=more.pop('splits', 1), epilogue=epi, a=a,
                                 lda=lda, stride_a=sa, b=b, ldb=ldb, stride_b=sb, c=c, ldc=ldc, stride_c=sc, **more)

    def _build_calls(self):
        G, B, P = self.G, self.B, self.P
        H, N = DIMS[1], DIMS[-1]
        lay = self.lay
        w16 = self.w16.data_ptr()
        par = self.params.data_ptr()
        grd = self.grad.data_ptr()
        bf, f4 = 2, 4
        fwd = []
        acts = [(self.x16, IN_PAD)] + [(h, H) for h in self.h]      # inputs of layers 1..4
        for layer in range(4):
            a, lda = acts[layer]
            o, rows, cols = lay['W%d' % layer]
            ob, _ = lay['b%d' % layer]
            common = (B, rows, cols, a.data_ptr(), lda, B * lda, w16 + o * bf, cols, P)
            if layer < 3:
                fwd.append(self._gemm(_abi.EPI_BIAS_SILU, *common, self.h[layer].data_ptr(), H, B * H,
                                      bias=par + ob * f4, stride_bias=P, c2=self.z[layer].data_ptr(), ldc2=H,
                                      stride_c2=B * H))
            else:
                # the output layer leaves the loss and its gradient; the outputs are not stored
                g = self.g16[3]
                fwd.append(self._gemm(_abi.EPI_LOSS, *common, g.data_ptr(), g.shape[2], B * g.shape[2],
                                      bias=par + ob * f4, stride_bias=P, aux=self.t.data_ptr(), ldaux=N,
                                      stride_aux=B * N, weights=self.w_out.data_ptr(), loss=self.loss.data_ptr(),
                                      c2=self.g32[3].data_ptr(), ldc2=g.shape[2], stride_c2=B * g.shape[2]))
        self.fwd_calls = fwd
        # G_{l-1} = (G_l W_l) * silu'(Z_{l-1}): A = G_l, B = W_l as it lies ([out, in])
        bwd = []
        for layer in (3, 2, 1):
            o, rows, cols = lay['W%d' % layer]
            g, prev = self.g16[layer], self.g16[layer - 1]
            bwd.append(self._gemm(_abi.EPI_DSILU, B, cols, rows, g.data_ptr(), g.shape[2], B * g.shape[2],
                                  w16 + o * bf, cols, P, prev.data_ptr(), H, B * H, trans_b=1,
                                  aux=self.z[layer - 1].data_ptr(), ldaux=H, stride_aux=B * H,
                                  c2=self.g32[layer - 1].data_ptr(), ldc2=H, stride_c2=B * H))
        self.bwd_calls = bwd
        # dW_l[o, i] = sum_b G[b, o] X[b, i] and db_l[o] = sum_b G[b, o], the four layers in one launch
        dw = (_abi.GemmProblemC * 4)()
        self.reduce_calls = []
        for layer in range(4):
            o, rows, cols = lay['W%d' % layer]
            ob, nb = lay['b%d' % layer]
            g = self.g16[layer]
            a, lda = acts[layer]
            c, sc, s_split = grd + o * f4, P, 0
            if self.splits > 1:
                part = self.part[layer]
                c, sc, s_split = part.data_ptr(), rows * cols, G * rows * cols
                self.reduce_calls.append((part.data_ptr(), s_split, sc, cols, grd + o * f4, P, cols, self.splits, G,
                                          rows, cols))
            dw[layer] = self._gemm(_abi.EPI_F32, rows, cols, B, g.data_ptr(), g.shape[2], B * g.shape[2],
                                   a.data_ptr(), lda, B * lda, c, cols, sc, splits=self.splits, stride_split=s_split,
                                   trans_a=1, trans_b=1, colsum=grd + ob * f4, stride_bias=P,
                                   colsum_in=self.g32[layer].data_ptr(), ld_colsum=g.shape[2],
                                   stride_colsum=B * g.shape[2], colsum_rows=self.colsum_rows)
        self.dw_calls = dw
        tb = (_abi.TransposeBlockC * 3)()
        for q, layer in enumerate((1, 2, 3)):
            o, rows, cols_ = lay['W%d' % layer]
            to, ld = self.tlay['W%d' % layer]
            tb[q] = _abi.TransposeBlockC(o, to, ld, rows, cols_)
        self.transpose_blocks = tb

    def _check(self, rc, what):
        if rc:
            raise _abi.McwError(rc, '%s failed' % what)

    def _launch(self, adam=True):
        """The kernels of one step on the current stream (no host synchronisation)."""
        L = _abi.load()
        st = _stream(self.torch)
        G, B = self.G, self.B
        N = DIMS[-1]
        self._check(L.mcw_mlp_step_begin(self.x_all.data_ptr(), self.t_all.data_ptr(), self.t_all.shape[1], N,
                                         self.perm.data_ptr(), self.n_rows, self.counter.data_ptr(), B, G,
                                         self.x16.data_ptr(), B * IN_PAD, self.t.data_ptr(), N, B * N,
                                         self.loss.data_ptr(), st), 'mcw_mlp_step_begin')
        for c in self.fwd_calls:
            self._check(L.mcw_mlp_gemm_batch(ctypes.byref(c), 1, st), 'forward product')
        for c in self.bwd_calls:
            self._check(L.mcw_mlp_gemm_batch(ctypes.byref(c), 1, st), 'backward product')
        self._check(L.mcw_mlp_gemm_batch(self.dw_calls, 4, st), 'weight gradients')
        for c in self.reduce_calls:
            self._check(L.mcw_mlp_reduce_splits(*c, st), 'mcw_mlp_reduce_splits')
        if not adam:
            return
        self._check(L.mcw_mlp_adam_grouped(self.params.data_ptr(), self.grad.data_ptr(), self.m.data_ptr(),
                                           self.v.data_ptr(), self.w16.data_ptr(), self.P, G, self.lr.data_ptr(),
                                           self.step.data_ptr(), self.beta1, self.beta2, self.eps,
                                           self.wt.data_ptr(), self.T, self.transpose_blocks, 3, st),
                    'mcw_mlp_adam_grouped')
        self._check(L.mcw_mlp_advance(self.counter.data_ptr(), self.step.data_ptr(), st), 'mcw_mlp_advance')

    def set_epoch(self, perms, lr):
        """Row order of each member for the next len(rows) // batch steps, and the learning rate."""
        torch = self.torch
        self.perm.copy_(torch.as_tensor(np.asarray(perms, np.int32)))
        self.counter.zero_()
        self.lr.fill_(float(lr))

    def run_step(self):
        """One Adam step of every member (graph replay after the first)."""
        torch = self.torch
        if not self.use_graph:
            self._launch()
            return
        if self.graph is None:
            # an eager step first: one-time set-up (module loading, kernel attributes)
            # must not happen inside the capture; then undo it
            saved = [t.clone() for t in (self.params, self.m, self.v, self.w16, self.wt, self.counter, self.step)]
            self._launch()
            for t, s0 in zip((self.params, self.m, self.v, self.w16, self.wt, self.counter, self.step), saved):
                t.copy_(s0)
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph):
                self._launch()
        self.graph.replay()

    def gradients(self):
        """Forward and backward of the current batch without the Adam step: the
        gradients of every member as [W1, b1, ..., W4, b4] (W1 without its padding)."""
        self._launch(adam=False)
        self.torch.cuda.synchronize()
        out = []
        for g in range(self.G):
            gr = []
            for layer in range(4):
                o, rows, cols = self.lay['W%d' % layer]
                w = self.grad[g, o:o + rows * cols].view(rows, cols)
                gr.append(w[:, :DIMS[layer]].clone())
                ob, nb = self.lay['b%d' % layer]
                gr.append(self.grad[g, ob:ob + nb].clone())
            out.append(gr)
        return out

    def export(self):
        """Copy the trained parameters, moments and step count back into the members."""
        torch = self.torch
        torch.cuda.synchronize()
        step = int(self.step.item()) - 1
        for g, net in enumerate(self.members):
            for layer in range(4):
                o, rows, cols = self.lay['W%d' % layer]
                k = DIMS[layer]
                for dst, src in ((net.params, self.params), (net.m, self.m), (net.v, self.v)):
                    dst[2 * layer].copy_(src[g, o:o + rows * cols].view(rows, cols)[:, :k])
                ob, nb = self.lay['b%d' % layer]
                for dst, src in ((net.params, self.params), (net.m, self.m), (net.v, self.v)):
                    dst[2 * layer + 1].copy_(src[g, ob:ob + nb])
            net.w16 = [_cast(torch, w.contiguous()) for w in net.params[0::2]]
            net.step = step
            net._blob = None


@dataclass
class Dataset:
    x: np.ndarray        # encoded inputs [n, 4]
    y: np.ndarray        # target space [n, 649]
    raw: np.ndarray      # (r_eff, wvl, mu0, depth) [n, 4]
    brf: np.ndarray      # [n, 648]
    albedo: np.ndarray   # [n]
    photons: int


def sample_inputs(n, seed):
    rng = np.random.default_rng(seed)
    r = np.exp(rng.uniform(np.log(R_RANGE[0]), np.log(R_RANGE[1]), n))
    wvl = rng.uniform(*WVL_RANGE, n)
    mu0 = rng.uniform(*MU_RANGE, n)
    depth = np.exp(rng.uniform(np.log(DEPTH_RANGE[0]), np.log(DEPTH_RANGE[1]), n))
    return np.stack([r, wvl, mu0, depth], axis=1)


def mc_brf(walker, raw, n_photon, seed, half_width=0.085, R=0.5, chunk=1024):
    """BRF (648 bins) and albedo of each input row by the GPU walk (n_photon photons each)."""
    from . import ssp
    from .config import WalkConfig
    raw = np.asarray(raw, np.float64)
    brf = np.zeros((raw.shape[0], N_BRF))
    alb = np.zeros(raw.shape[0])
    imp = ssp.synthetic_impurity_table(600, 2100)
    for lo in range(0, raw.shape[0], chunk):
        rows = raw[lo:lo + chunk]
        tables, cfgs = [], []
        for j, (r, wvl, mu0, depth) in enumerate(rows):
            tables.append(ssp.synthetic_ice_table(r, 600, 2100))
            tau = depth * ssp.ext_cff_mss_sphere(r) * 300.0
            theta0 = math.degrees(math.acos(min(1.0, max(0.0, mu0))))
            cfgs.append(WalkConfig(n_photon=int(n_photon), wvl0=float(wvl), half_width=half_width,
                                   theta0_deg=min(theta0, 89.999), tau_tot=tau,
                                   lambertian_reflectance=R, ice_table=j, rds_snw=float(r)))
        walker.set_tables(tables, imp)
        res = walker.walk(cfgs, seed + lo, mode='f32', records=None)
        b, a = res.brf()
        brf[lo:lo + len(rows)] = b
        alb[lo:lo + len(rows)] = a
    return brf, alb


class Ensemble:
    """Members trained on the same data from different initialisations and batch orders."""

    def __init__(self, members):
        self.members = members
        self._pack = None         # (key, blob of every member's packed weights, their biases)

    def packed(self):
        """The members' packed weights one after the other and their biases as rows
        (float32 [members, 1417]), rebuilt when any member's weights change."""
        import torch
        key = tuple((m.step, tuple(w.data_ptr() for w in m.w16), tuple(b.data_ptr() for b in m.params[1::2]))
                    for m in self.members)
        if self._pack is None or self._pack[0] != key:
            blob = torch.cat([m.packed() for m in self.members])
            bias = torch.stack([torch.cat([b.float().reshape(-1) for b in m.params[1::2]]) for m in self.members])
            self._pack = (key, blob, bias.contiguous())
        return self._pack[1], self._pack[2]

    def predict_std(self, x):
        """Every member's standardised outputs for encoded inputs x (torch CUDA float32
        [n, 4]) in one launch of the fused kernel: fp16 [members, n, 649]."""
        import torch
        blob, bias = self.packed()
        return forward_ensemble(torch, x, blob, bias, len(self.members))

    def scaling(self):
        """The members' target scaling as rows: (mean, std), float64 [members, 649]."""
        import torch
        return (torch.stack([m.y_mean.double() for m in self.members]).contiguous(),
                torch.stack([m.y_std.double() for m in self.members]).contiguous())

    def member_brfs(self, x):
        """Each member's BRF [members, n, 648] and albedo [members, n] (torch CUDA float64) for
        encoded inputs x (torch CUDA float32 [n, 4])."""
        return self._member_brfs(x, *self.scaling())

    def _member_brfs(self, x, mean, std):
        import torch
        ys = self.predict_std(x)
        k, n = ys.shape[:2]
        brf = torch.empty((k, n, N_BRF), dtype=torch.float64, device=x.device)
        alb = torch.empty((k, n), dtype=torch.float64, device=x.device)
        rc = _abi.load().mcw_brf_members(_ptr(ys), ys.stride(1), k, n, _ptr(mean), _ptr(std), BRF_FLOOR, _ptr(brf),
                                         _ptr(alb), _stream(torch))
        if rc:
            raise _abi.McwError(rc, 'mcw_brf_members failed')
        return brf, alb

    def brf_stats(self, brf, alb):
        """Mean BRF [n, 648], mean albedo [n] and relative spread [n] of member_brfs' result
        (torch CUDA float64): the spread in the units of rel_rms, weighted RMS standard
        deviation over weighted RMS BRF."""
        import torch
        return self._brf_stats(brf, alb, torch.from_numpy(bin_weights()).to(brf.device))

    def _brf_stats(self, brf, alb, share):
        import torch
        k, n = alb.shape
        mean = torch.empty((n, N_BRF), dtype=torch.float64, device=brf.device)
        alb_mean, spread = torch.empty_like(alb[0]), torch.empty_like(alb[0])
        rc = _abi.load().mcw_brf_stats(_ptr(brf), _ptr(alb), k, n, _ptr(share), _ptr(mean), _ptr(alb_mean),
                                       _ptr(spread), _stream(torch))
        if rc:
            raise _abi.McwError(rc, 'mcw_brf_stats failed')
        return mean, alb_mean, spread

    def _chunks(self, raw, rows=16384):
        import torch
        x = encode(*np.asarray(raw, np.float64).T)
        for lo in range(0, x.shape[0], rows):
            yield torch.from_numpy(x[lo:lo + rows]).cuda()

    def predict_members(self, raw):
        """Each member's BRF [members, n, 648] and albedo [members, n]."""
        parts = [[t.cpu().numpy() for t in self.member_brfs(x)] for x in self._chunks(raw)]
        if not parts:
            k = len(self.members)
            return np.zeros((k, 0, N_BRF)), np.zeros((k, 0))
        return np.concatenate([p[0] for p in parts], 1), np.concatenate([p[1] for p in parts], 1)

    def predict(self, raw):
        """Mean BRF [n, 648], mean albedo [n], relative ensemble spread of the BRF [n]."""
        parts = [[t.cpu().numpy() for t in self.brf_stats(*self.member_brfs(x))] for x in self._chunks(raw)]
        if not parts:
            return np.zeros((0, N_BRF)), np.zeros(0), np.zeros(0)
        return tuple(np.concatenate([p[k] for p in parts]) for k in range(3))


def bin_weights():
    """Solid-angle weights sin(theta) cos(theta) of the 648 bins (the expected photon share)."""
    mids = (np.arange(18) + 0.5) * (np.pi / 36)
    w = np.sin(mids) * np.cos(mids)
    return np.repeat(w / w.sum() / 36, 36)


def rel_rms(pred, ref, weights=None):
    """RMS relative BRF error per config: sqrt(sum_b w_b (pred - ref)^2 / sum_b w_b ref^2),
    bins weighted by their solid-angle share w_b (the photons they receive)."""
    w = bin_weights() if weights is None else weights
    return np.sqrt(((pred - ref) ** 2 * w).sum(axis=-1) / np.maximum((ref ** 2 * w).sum(axis=-1), 1e-30))


def train(ds, members=5, epochs=400, batch=256, lr=1e-3, seed=0, log=None, engine='grouped'):
    """Train an ensemble on a Dataset; returns Ensemble.  engine 'grouped': all members
    at once on the training engine (EnsembleTrainer, one graph replay per step);
    'layerwise': member by member on mcw_mlp_gemm and the per-member kernels."""
    import torch
    y = ds.y.astype(np.float64)
    y_mean, y_std = y.mean(0), np.maximum(y.std(0), 1e-3)
    t_all = torch.from_numpy(((y - y_mean) / y_std).astype(np.float32)).cuda()
    x_all = _cast(torch, torch.from_numpy(ds.x).cuda())
    w_out = torch.from_numpy(output_weights()).cuda()
    n = ds.x.shape[0]
    nets = []
    for k in range(members):
        net = SurrogateMLP(seed=seed * 100 + k)
        net.y_mean = torch.from_numpy(y_mean).cuda()
        net.y_std = torch.from_numpy(y_std).cuda()
        nets.append(net)
    if engine == 'grouped':
        # every member's step in one captured graph of grouped launches
        rngs = [np.random.default_rng(seed * 100 + k) for k in range(members)]
        tr = EnsembleTrainer(nets, batch, torch.from_numpy(ds.x).cuda(), t_all, w_out, lr=lr)
        for ep in range(epochs):
            lr_ep = lr * (0.5 * (1 + math.cos(math.pi * ep / epochs)))
            tr.set_epoch([r.permutation(n) for r in rngs], lr_ep)
            for _ in range(n // batch):
                tr.run_step()
            if log and (ep % 50 == 0 or ep == epochs - 1):
                log('epoch %d loss %s' % (ep, np.round(tr.loss.cpu().numpy(), 5).tolist()))
        tr.export()
        return Ensemble(nets)
    for k, net in enumerate(nets):
        rng = np.random.default_rng(seed * 100 + k)
        for ep in range(epochs):
            perm = torch.from_numpy(rng.permutation(n)).cuda()
            lr_ep = lr * (0.5 * (1 + math.cos(math.pi * ep / epochs)))
            for lo in range(0, n - batch + 1, batch):
                idx = perm[lo:lo + batch]
                loss = net.train_step(x_all[idx].contiguous(), t_all[idx].contiguous(), w_out, lr=lr_ep)
            if log and (ep % 50 == 0 or ep == epochs - 1):
                log('member %d epoch %d loss %.5f' % (k, ep, float(loss)))
    torch.cuda.synchronize()
    return Ensemble(nets)


def save(ensemble, path):
    """FP32 master weights, Adam state and target scaling of every member (torch.save)."""
    import torch
    torch.save([{'params': [p.cpu() for p in m.params], 'm': [x.cpu() for x in m.m],
                 'v': [x.cpu() for x in m.v], 'step': m.step, 'y_mean': m.y_mean.cpu(),
                 'y_std': m.y_std.cpu()} for m in ensemble.members], path)


def load(path):
    import torch
    members = []
    for d in torch.load(path):
        net = SurrogateMLP()
        net.params = [p.cuda() for p in d['params']]
        net.m = [x.cuda() for x in d['m']]
        net.v = [x.cuda() for x in d['v']]
        net.w16 = [_cast(torch, w) for w in net.params[0::2]]
        net.step = d['step']
        net.y_mean, net.y_std = d['y_mean'].cuda(), d['y_std'].cuda()
        members.append(net)
    return Ensemble(members)


def make_dataset(walker, n_cfg, n_photon, seed):
    raw = sample_inputs(n_cfg, seed)
    brf, alb = mc_brf(walker, raw, n_photon, seed)
    x = encode(*raw.T)
    return Dataset(x=x, y=to_target(brf, alb), raw=raw, brf=brf, albedo=alb, photons=n_photon)


def output_weights():
    """Loss weights: BRF bins by their photon share (mean 1), albedo 10."""
    w = bin_weights()
    w = w / w.mean()
    return np.concatenate([w, [10.0]]).astype(np.float32)


def inference_rate(ensemble, batch=65536, reps=20, members=None):
    """BRF predictions per second on the fused tensor-core kernel (CUDA events): every member
    of the ensemble (the mean and spread of a prediction need them all) forwards the same
    batch in one launch (mcw_mlp_forward_ensemble_f16); with members=k, the first k members
    one launch each.  The L2 is flushed before each timed repetition (median over reps)."""
    import torch
    ms = ensemble.members if members is None else ensemble.members[:members]
    x = torch.rand((batch, 4), device='cuda') * 2 - 1
    run = ensemble.predict_std if members is None else (lambda v: [m.predict_std(v) for m in ms])
    for _ in range(3):
        run(x)
    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device='cuda')
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(reps):
        flush.zero_()
        e0.record()
        run(x)
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    del flush
    return batch / (float(np.median(times)) / 1e3)
