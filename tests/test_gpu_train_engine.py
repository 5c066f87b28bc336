"""The surrogate's training engine on the GPU (include/mcw_mlp.h, EnsembleTrainer):
the grouped TMA-fed tcgen05 GEMM against float64 on the same bf16 operands (every
epilogue, groups, split-K, transposed copies), one ensemble step's gradients against
float64 CPU autograd of each member, the grouped Adam against its formula, the
captured step against the same step run eagerly, and training that converges."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from monte_carlompi_gb300 import _abi, surrogate  # noqa: E402
from tests.helpers import reference_mlp  # noqa: E402


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _status_clear():
    flags = ctypes.c_uint32(0)
    assert _abi.load().mcw_mlp_status(1, ctypes.byref(flags)) == 0


def _status_ok():
    flags = ctypes.c_uint32(0)
    assert _abi.load().mcw_mlp_status(0, ctypes.byref(flags)) == 0
    assert flags.value == 0, flags.value


def _grouped(epi, m, n, k, a, b, c, groups=1, splits=1, bias=None, aux=None, c2=None, ct=None, s_split=0):
    """a [G, m, lda], b [G, n, ldb] bf16; c [G, m, ldc] (split partials: [S, G, m, ldc])."""
    lda, ldb = a.shape[-1], b.shape[-1]
    ldc = c.shape[-1]
    p = _abi.GemmGroupedC(m, n, k, groups, splits, epi, a.data_ptr(), lda, a.shape[-2] * lda,
                          b.data_ptr(), ldb, b.shape[-2] * ldb,
                          bias.data_ptr() if bias is not None else None, bias.shape[-1] if bias is not None else 0,
                          aux.data_ptr() if aux is not None else None, aux.shape[-1] if aux is not None else 0,
                          aux.shape[-2] * aux.shape[-1] if aux is not None else 0,
                          c.data_ptr(), ldc, c.shape[-2] * ldc, s_split,
                          c2.data_ptr() if c2 is not None else None, c2.shape[-1] if c2 is not None else 0,
                          c2.shape[-2] * c2.shape[-1] if c2 is not None else 0,
                          ct.data_ptr() if ct is not None else None, ct.shape[-1] if ct is not None else 0,
                          ct.shape[-2] * ct.shape[-1] if ct is not None else 0)
    return _abi.load().mcw_mlp_gemm_grouped(ctypes.byref(p), _stream())


@pytest.mark.parametrize('m,n,k,groups', [(128, 128, 64, 1), (300, 200, 256, 3), (256, 649, 256, 5),
                                          (1000, 256, 16, 2), (77, 40, 1000, 2), (649, 256, 4096, 1)])
def test_grouped_gemm_matches_float64(m, n, k, groups):
    g = torch.Generator().manual_seed(m + n + k + groups)
    ka = (k + 7) // 8 * 8
    a = torch.zeros(groups, m, ka)
    b = torch.zeros(groups, n, ka)
    a[:, :, :k] = torch.randn(groups, m, k, generator=g)
    b[:, :, :k] = torch.randn(groups, n, k, generator=g) * 0.1
    a16, b16 = a.to(torch.bfloat16).cuda(), b.to(torch.bfloat16).cuda()
    c = torch.full((groups, m, n), 7.0, device='cuda')
    _status_clear()
    assert _grouped(_abi.EPI_F32, m, n, k, a16, b16, c, groups=groups) == 0
    torch.cuda.synchronize()
    _status_ok()
    ref = a16.cpu().double()[:, :, :k] @ b16.cpu().double()[:, :, :k].transpose(1, 2)
    err = (c.cpu().double() - ref).abs().max().item()
    assert err <= 1e-4 * max(1.0, ref.abs().max().item()) + 1e-5 * math.sqrt(k), err


def test_grouped_gemm_split_k_partials_add_up():
    """K = 4,096 cut into 4 ranges: the partial products add up to the whole product."""
    groups, m, n, k, splits = 2, 300, 256, 4096, 4
    g = torch.Generator().manual_seed(3)
    a16 = torch.randn(groups, m, k, generator=g).to(torch.bfloat16).cuda()
    b16 = (torch.randn(groups, n, k, generator=g) * 0.1).to(torch.bfloat16).cuda()
    part = torch.zeros(splits, groups, m, n, device='cuda')
    assert _grouped(_abi.EPI_F32, m, n, k, a16, b16, part, groups=groups, splits=splits,
                    s_split=groups * m * n) == 0
    out = torch.zeros(groups, m, n, device='cuda')
    rc = _abi.load().mcw_mlp_reduce_splits(part.data_ptr(), groups * m * n, m * n, n, out.data_ptr(), m * n, n,
                                           splits, groups, m, n, _stream())
    assert rc == 0
    torch.cuda.synchronize()
    ref = a16.cpu().double() @ b16.cpu().double().transpose(1, 2)
    assert (out.cpu().double() - ref).abs().max().item() < 1e-4 * ref.abs().max().item()
    # a split count the K range cannot be cut into (64 chunks: 9 splits of 8 chunks are 8) is refused
    assert _grouped(_abi.EPI_F32, m, n, k, a16, b16, part, groups=groups, splits=9, s_split=groups * m * n) == -1


def test_grouped_gemm_epilogues_and_transposed_copies():
    groups, m, n, k = 3, 200, 256, 256
    g = torch.Generator().manual_seed(9)
    a16 = torch.randn(groups, m, k, generator=g).to(torch.bfloat16).cuda()
    w16 = (torch.randn(groups, n, k, generator=g) * 0.1).to(torch.bfloat16).cuda()
    bias = torch.randn(groups, n, generator=g).cuda()
    act = torch.zeros(groups, m, n, dtype=torch.bfloat16, device='cuda')
    z = torch.zeros(groups, m, n, device='cuda')
    act_t = torch.zeros(groups, n, m, dtype=torch.bfloat16, device='cuda')
    assert _grouped(_abi.EPI_BIAS_SILU, m, n, k, a16, w16, act, groups=groups, bias=bias, c2=z, ct=act_t) == 0
    torch.cuda.synchronize()
    zr = a16.cpu().double() @ w16.cpu().double().transpose(1, 2) + bias.cpu().double()[:, None, :]
    assert (z.cpu().double() - zr).abs().max().item() < 1e-4 * zr.abs().max().item()
    sr = zr * torch.sigmoid(zr)
    assert (act.cpu().double() - sr).abs().max().item() <= 0.01 * sr.abs().max().item()
    assert torch.equal(act_t.cpu(), act.cpu().transpose(1, 2))
    # SiLU' product with its copies
    gout = torch.zeros(groups, m, n, dtype=torch.bfloat16, device='cuda')
    g32 = torch.zeros(groups, m, n, device='cuda')
    gt = torch.zeros(groups, n, m, dtype=torch.bfloat16, device='cuda')
    assert _grouped(_abi.EPI_DSILU, m, n, k, a16, w16, gout, groups=groups, aux=z, c2=g32, ct=gt) == 0
    torch.cuda.synchronize()
    s = torch.sigmoid(z.cpu().double())
    gr = (a16.cpu().double() @ w16.cpu().double().transpose(1, 2)) * s * (1 + z.cpu().double() * (1 - s))
    assert (g32.cpu().double() - gr).abs().max().item() < 1e-3 * gr.abs().max().item()
    assert torch.equal(gt.cpu(), gout.cpu().transpose(1, 2))
    assert torch.equal(gout.cpu(), g32.cpu().to(torch.bfloat16))


def test_grouped_gemm_refuses_operands_tma_cannot_copy():
    a16 = torch.zeros(1, 64, 20, dtype=torch.bfloat16, device='cuda')      # rows of 40 bytes
    b16 = torch.zeros(1, 64, 24, dtype=torch.bfloat16, device='cuda')
    c = torch.zeros(1, 64, 64, device='cuda')
    assert _grouped(_abi.EPI_F32, 64, 64, 20, a16, b16, c) == -1
    flat = torch.zeros(64 * 24 + 4, dtype=torch.bfloat16, device='cuda')
    off = flat[4:].view(1, 64, 24)                                          # 8-byte aligned base
    assert _grouped(_abi.EPI_F32, 64, 64, 24, off, b16, c) == -1


def _members(n, seed):
    nets = [surrogate.SurrogateMLP(seed=seed + k) for k in range(n)]
    g = torch.Generator().manual_seed(seed)
    for net in nets:                                    # non-zero biases
        for i in range(1, 8, 2):
            net.params[i].copy_((torch.randn(net.params[i].shape, generator=g) * 0.3).cuda())
        net.w16 = [surrogate._cast(torch, w) for w in net.params[0::2]]
    return nets


def _data(n_rows, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.rand(n_rows, 4, generator=g) * 2 - 1
    t = torch.randn(n_rows, 649, generator=g)
    w = torch.from_numpy(surrogate.output_weights())
    return x, t, w


@pytest.mark.parametrize('batch,n_rows', [(256, 1024), (4096, 4096)])
def test_ensemble_gradients_match_cpu_autograd(batch, n_rows):
    """Forward, loss and backward of three members on their own batches (one launch per
    product for all members; at 4,096 rows the weight gradients are split-K) against
    float64 CPU autograd of each member (same bf16 roundings of weights, inputs and
    activations)."""
    nets = _members(3, 50)
    x, t, w = _data(n_rows, 4)
    tr = surrogate.EnsembleTrainer(nets, batch, x.cuda(), t.cuda(), w.cuda(), use_graph=False)
    rng = np.random.default_rng(1)
    perms = [rng.permutation(n_rows) for _ in nets]
    tr.set_epoch(perms, 1e-3)
    _status_clear()
    grads = tr.gradients()
    _status_ok()
    for k, net in enumerate(nets):
        idx = torch.from_numpy(perms[k][:batch])
        params = [p.detach().cpu().double().requires_grad_(True) for p in net.params]
        xb = x[idx].double()
        y = reference_mlp(xb, params)
        d = y - t[idx].double()
        loss = (w.double() * d * d).sum() / (batch * 649)
        loss.backward()
        assert abs(float(tr.loss[k]) - loss.item()) < 1e-3 * loss.item()
        for got, ref in zip(grads[k], params):
            got = got.cpu().double().flatten()
            ref = ref.grad.flatten()
            rel = (got - ref).norm() / ref.norm()
            cos = torch.dot(got, ref) / (got.norm() * ref.norm())
            assert rel < 3e-2 and cos > 0.999, (k, rel.item(), cos.item())


def test_ensemble_adam_matches_formula_and_graph_matches_eager():
    """Three captured steps equal three eager steps bit for bit; one step's update equals
    Adam's formula on the gradients the engine computed."""
    x, t, w = _data(1024, 6)
    rng = np.random.default_rng(2)
    perms = [rng.permutation(1024) for _ in range(2)]
    a = surrogate.EnsembleTrainer(_members(2, 70), 256, x.cuda(), t.cuda(), w.cuda(), use_graph=True)
    b = surrogate.EnsembleTrainer(_members(2, 70), 256, x.cuda(), t.cuda(), w.cuda(), use_graph=False)
    for tr in (a, b):
        tr.set_epoch(perms, 2e-3)
        for _ in range(3):
            tr.run_step()
    torch.cuda.synchronize()
    assert torch.equal(a.params, b.params) and torch.equal(a.m, b.m) and torch.equal(a.v, b.v)
    assert torch.equal(a.w16, b.w16) and torch.equal(a.wt, b.wt)
    assert int(a.step.item()) == 4 and int(a.counter.item()) == 3
    # one more step on b, checked against the formula
    w0, m0, v0 = b.params.clone(), b.m.clone(), b.v.clone()
    grads = b.gradients()            # the gradients of the next batch (counter 3)
    flat = b.grad.clone()
    b.run_step()
    torch.cuda.synchronize()
    lr, b1, b2, eps, step = 2e-3, 0.9, 0.999, 1e-8, 4
    m1 = b1 * m0 + (1 - b1) * flat
    v1 = b2 * v0 + (1 - b2) * flat * flat
    w1 = w0 - lr * (m1 / (1 - b1 ** step)) / (torch.sqrt(v1 / (1 - b2 ** step)) + eps)
    assert torch.allclose(b.params, w1, atol=1e-6, rtol=1e-5)
    assert torch.equal(b.w16, b.params.to(torch.bfloat16))
    o, rows, cols = b.lay['W3']
    to, ld = b.tlay['W3']
    wt = b.wt[:, to:to + cols * ld].view(2, cols, ld)
    assert torch.equal(wt[:, :, :rows], b.w16[:, o:o + rows * cols].view(2, rows, cols).transpose(1, 2))
    assert (wt[:, :, rows:] == 0).all()
    assert len(grads) == 2 and grads[0][6].shape == (649, 256)


def test_ensemble_training_fits_a_smooth_map():
    """Two members trained together on a smooth 4 -> 649 map: each member's loss falls a
    hundredfold, and the exported networks predict through the fused inference kernel."""
    rng = np.random.default_rng(0)
    n = 2048
    x = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    basis = rng.standard_normal((4, 649)) * 0.7
    y = np.tanh(x @ basis) + 0.3 * np.sin(2 * x[:, :1])
    y = ((y - y.mean(0)) / y.std(0)).astype(np.float32)
    nets = [surrogate.SurrogateMLP(seed=1 + k) for k in range(2)]
    tr = surrogate.EnsembleTrainer(nets, 256, torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(),
                                   torch.ones(649, device='cuda'), lr=2e-3)
    first = None
    for ep in range(120):
        tr.set_epoch([rng.permutation(n) for _ in nets], 2e-3)
        for _ in range(n // 256):
            tr.run_step()
        if first is None:
            torch.cuda.synchronize()
            first = tr.loss.cpu().numpy().copy()
    last = tr.loss.cpu().numpy()
    assert np.all(last < first / 100), (first, last)
    tr.export()
    xt = torch.from_numpy(x[:512]).cuda()
    for net in nets:
        pred = net.predict_std(xt, half=False)
        err = ((pred - torch.from_numpy(y[:512]).cuda()) ** 2).mean().item()
        assert err < 0.05, err


def _problem(epi, m, n, k, a, b, c, ta, tb, groups=1, **more):
    f = dict(m=m, n=n, k=k, groups=groups, splits=1, epilogue=epi, trans_a=ta, trans_b=tb, a=a.data_ptr(),
             lda=a.shape[-1], stride_a=a.shape[-2] * a.shape[-1], b=b.data_ptr(), ldb=b.shape[-1],
             stride_b=b.shape[-2] * b.shape[-1], c=c.data_ptr(), ldc=c.shape[-1],
             stride_c=c.shape[-2] * c.shape[-1])
    f.update(more)
    return _abi.GemmProblemC(**f)


@pytest.mark.parametrize('ta,tb', [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize('m,n,k', [(1, 1, 1), (129, 33, 63), (128, 64, 65), (40000, 65, 17), (255, 4, 1000)])
def test_gemm_batch_layouts_match_float64(ta, tb, m, n, k):
    """Operands stored along either dimension, remainders of every tile, two groups, and two
    problems of different sizes in one launch."""
    g = torch.Generator().manual_seed(m + 7 * n + 11 * k + ta + 2 * tb)
    r8 = lambda v: (v + 7) // 8 * 8  # noqa: E731
    calls = (_abi.GemmProblemC * 2)()
    keep = []
    for i, (mm, nn, kk) in enumerate(((m, n, k), (n, m if m < 3000 else 9, k + 5))):
        a = torch.randn((2, kk, r8(mm)) if ta else (2, mm, r8(kk)), generator=g).to(torch.bfloat16).cuda()
        b = (torch.randn((2, kk, r8(nn)) if tb else (2, nn, r8(kk)), generator=g) * 0.1).to(torch.bfloat16).cuda()
        c = torch.full((2, mm + 1, nn + 1), 7.0, device='cuda')        # a row and a column that stay
        calls[i] = _problem(_abi.EPI_F32, mm, nn, kk, a, b, c, ta, tb, groups=2)
        keep.append((a, b, c, mm, nn, kk))
    _status_clear()
    assert _abi.load().mcw_mlp_gemm_batch(calls, 2, _stream()) == 0
    torch.cuda.synchronize()
    _status_ok()
    for a, b, c, mm, nn, kk in keep:
        A = (a[:, :, :mm].transpose(1, 2) if ta else a[:, :, :kk]).cpu().double()
        B = (b[:, :, :nn] if tb else b[:, :, :kk].transpose(1, 2)).cpu().double()
        ref = A @ B
        err = (c[:, :mm, :nn].cpu().double() - ref).abs().max().item()
        assert err <= 1e-4 * max(1.0, ref.abs().max().item()) + 1e-5 * math.sqrt(kk), err
        assert (c[:, mm] == 7).all() and (c[:, :, nn] == 7).all()


@pytest.mark.parametrize('k', [2047, 2048, 2049, 2112, 2113, 4200])
def test_gemm_batch_long_chain_matches_float64(k):
    """A transposed product of few tiles and a long K, two chunks of 64 a stage: a last stage of
    one chunk, chunks cut short, and more stages than the ring holds."""
    m, n = 200, 72
    g = torch.Generator().manual_seed(k)
    a = torch.randn((2, k, m), generator=g).to(torch.bfloat16).cuda()
    b = (torch.randn((2, k, n), generator=g) * 0.1).to(torch.bfloat16).cuda()
    c = torch.full((2, m + 1, n + 1), 7.0, device='cuda')
    q = _problem(_abi.EPI_F32, m, n, k, a, b, c, 1, 1, groups=2)
    _status_clear()
    assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
    torch.cuda.synchronize()
    _status_ok()
    ref = a.cpu().double().transpose(1, 2) @ b.cpu().double()
    err = (c[:, :m, :n].cpu().double() - ref).abs().max().item()
    assert err <= 1e-4 * max(1.0, ref.abs().max().item()) + 1e-5 * math.sqrt(k), err
    assert (c[:, m] == 7).all() and (c[:, :, n] == 7).all()


@pytest.mark.parametrize('m,n', [(128, 64), (31, 33), (640, 649)])
def test_silu_derivative_over_the_range(m, n):
    """The SiLU' epilogue from pre-activations of -100 to 100, infinities and NaN against float64:
    exp's argument is rounded at |z| 2^-23, the rest to a few units of 2^-24, and the sigmoid is 0
    where exp(-z) leaves FP32's range."""
    a = torch.ones(1, m, 8, dtype=torch.bfloat16, device='cuda') / 8
    b = torch.ones(1, n, 8, dtype=torch.bfloat16, device='cuda')
    z = torch.linspace(-100, 100, m * n).reshape(m, n)
    z[0, 0], z[0, 1], z[1, 0] = float('nan'), float('inf'), float('-inf')
    z[1, 1], z[2, 2] = 0.0, -88.0
    zc = z.cuda()
    out16 = torch.zeros(1, m, n, dtype=torch.bfloat16, device='cuda')
    out32 = torch.zeros(1, m, n, device='cuda')
    q = _problem(_abi.EPI_DSILU, m, n, 8, a, b, out16, 0, 0, aux=zc.data_ptr(), ldaux=n, stride_aux=m * n,
                 c2=out32.data_ptr(), ldc2=n, stride_c2=m * n)
    assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
    torch.cuda.synchronize()
    got = out32[0].cpu().double()
    zd = z.double()
    s = torch.where(torch.exp(-zd) > 3.4028235e38, 0.0, torch.sigmoid(zd))
    ref = s * (1 + zd * (1 - s))
    tol = 2e-5 * s * (1 + zd.abs()) + 1e-37
    odd = ~torch.isfinite(zd)
    assert (((got - ref).abs() <= tol) | odd).all()
    assert torch.isnan(got[0, 0]) and torch.isnan(got[1, 0])
    assert torch.equal(out16.float(), out32.to(torch.bfloat16).float()) or torch.isnan(out32).any()


@pytest.mark.parametrize('m,n', [(1, 649), (130, 40), (700, 256)])
def test_gemm_batch_loss_and_column_sums(m, n):
    """The loss epilogue, the column sums of SiLU' and loss results over every 128 rows, their
    total beside a plain product, and rows cast to padded bf16 with their column sums."""
    G, k = 2, 256
    g = torch.Generator().manual_seed(m + n)
    a = torch.randn(G, m, k, generator=g).to(torch.bfloat16).cuda()
    b = (torch.randn(G, n, k, generator=g) * 0.1).to(torch.bfloat16).cuda()
    aux = torch.randn(G, m, n, generator=g).cuda()
    bias, w = torch.randn(G, n, generator=g).cuda(), torch.rand(n, generator=g).cuda()
    blocks = (m + 127) // 128
    acc = a.cpu().double() @ b.cpu().double().transpose(1, 2)
    for epi in (_abi.EPI_LOSS, _abi.EPI_DSILU):
        out16 = torch.zeros(G, m, n, dtype=torch.bfloat16, device='cuda')
        out32 = torch.zeros(G, m, n, device='cuda')
        sums = torch.zeros(G, blocks, n, device='cuda')
        loss = torch.zeros(G, device='cuda')
        q = _problem(epi, m, n, k, a, b, out16, 0, 0, groups=G, aux=aux.data_ptr(), ldaux=n, stride_aux=m * n,
                     bias=bias.data_ptr(), stride_bias=n, c2=out32.data_ptr(), ldc2=n, stride_c2=m * n,
                     colsum=sums.data_ptr(), ld_colsum=n, stride_colsum=blocks * n, weights=w.data_ptr(),
                     loss=loss.data_ptr())
        assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
        torch.cuda.synchronize()
        x = aux.cpu().double()
        if epi == _abi.EPI_LOSS:
            d = acc + bias.cpu().double()[:, None] - x
            ref = 2 * w.cpu().double() * d / (m * n)
            lref = (w.cpu().double() * d * d).sum((1, 2)) / (m * n)
            assert ((loss.cpu().double() - lref).abs() < 1e-5 * lref).all()
        else:
            s = torch.sigmoid(x)
            ref = acc * s * (1 + x * (1 - s))
        assert (out32.cpu().double() - ref).abs().max() < 1e-4 * ref.abs().max()
        assert torch.equal(out16, out32.to(torch.bfloat16))
        for q0 in range(blocks):
            part = out32[:, 128 * q0:128 * q0 + 128].double().sum(1)
            assert (sums[:, q0].double() - part).abs().max() < 1e-5 * part.abs().max() + 1e-12
    # the total of the last sums beside the product it is the bias gradient of
    gt = torch.zeros(G, m, (n + 7) // 8 * 8, dtype=torch.bfloat16, device='cuda')
    gt[:, :, :n] = out16
    dw, db = torch.zeros(G, n, k, device='cuda'), torch.zeros(G, n, device='cuda')
    q = _problem(_abi.EPI_F32, n, k, m, gt, a, dw, 1, 1, groups=G, colsum=db.data_ptr(), stride_bias=n,
                 colsum_in=sums.data_ptr(), ld_colsum=n, stride_colsum=blocks * n, colsum_chunks=blocks)
    assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
    torch.cuda.synchronize()
    assert (db.double() - out32.double().sum(1)).abs().max() < 1e-5 * out32.double().sum(1).abs().max() + 1e-12
    ref = out16.cpu().double().transpose(1, 2) @ a.cpu().double()
    assert (dw.cpu().double() - ref).abs().max() < 1e-4 * ref.abs().max()
    # and from the rows themselves, in mcw_mlp_colsum_grouped's order, for any number of column tiles
    for rows in (m, 64, 1024):
        for kk in (k, 40, 100):
            one, two = torch.zeros(G, n, device='cuda'), torch.zeros(G, n, device='cuda')
            dw = torch.zeros(G, n, kk, device='cuda')
            x = a[:, :, :(kk + 7) // 8 * 8].contiguous()
            q = _problem(_abi.EPI_F32, n, kk, m, gt, x, dw, 1, 1, groups=G, colsum=one.data_ptr(), stride_bias=n,
                         colsum_in=out32.data_ptr(), ld_colsum=n, stride_colsum=m * n, colsum_rows=rows)
            assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
            layer = _abi.ColsumLayerC(out32.data_ptr(), n, m * n, 0, n, 0)
            part = torch.zeros(G * ((m + rows - 1) // rows) * n, device='cuda')
            assert _abi.load().mcw_mlp_colsum_grouped(ctypes.byref(layer), 1, G, m, two.data_ptr(), n,
                                                      part.data_ptr(), rows, _stream()) == 0
            torch.cuda.synchronize()
            assert torch.equal(one, two), (rows, kk)
    # padded rows
    src = out32[0].contiguous()
    dst = torch.full((m, (n + 7) // 8 * 8), 5.0, dtype=torch.bfloat16, device='cuda')
    cs = torch.zeros(blocks, n, device='cuda')
    rc = _abi.load().mcw_mlp_cast_rows(src.data_ptr(), 0, m, n, n, dst.data_ptr(), dst.shape[1], cs.data_ptr(), n,
                                       _stream())
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(dst[:, :n], src.to(torch.bfloat16)) and (dst[:, n:] == 0).all()
    assert (cs.double().sum(0) - src.double().sum(0)).abs().max() < 1e-5 * src.double().sum(0).abs().max() + 1e-12


@pytest.mark.parametrize('rows,ld', [(1, 8), (12, 16), (31, 40), (32, 32), (33, 48), (649, 656)])
def test_grouped_adam_writes_no_padding_of_the_transposed_copies(rows, ld):
    """wt[offset_t + c ld_t + o] is written for o < rows alone: what lies between the columns' ends,
    and behind the last column's, keeps what the caller had there."""
    G, cols = 2, 72
    n = rows * cols + 16
    off_t, stride_t = 8, 8 + (cols - 1) * ld + rows + 24
    stride_t += -stride_t % 8
    g = torch.Generator().manual_seed(rows)
    w, gr = torch.randn(G, n, generator=g).cuda(), torch.randn(G, n, generator=g).cuda()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    w16 = torch.zeros(G, n, dtype=torch.bfloat16, device='cuda')
    wt = torch.full((G, stride_t), 7.0, dtype=torch.bfloat16, device='cuda')
    lr, step = torch.full((1,), 1e-3, device='cuda'), torch.ones(1, dtype=torch.int32, device='cuda')
    blk = (_abi.TransposeBlockC * 1)(_abi.TransposeBlockC(8, off_t, ld, rows, cols))
    assert _abi.load().mcw_mlp_adam_grouped(w.data_ptr(), gr.data_ptr(), m.data_ptr(), v.data_ptr(), w16.data_ptr(), n, G,
                                            lr.data_ptr(), step.data_ptr(), 0.9, 0.999, 1e-8, wt.data_ptr(), stride_t,
                                            blk, 1, _stream()) == 0
    torch.cuda.synchronize()
    assert torch.equal(w16, w.to(torch.bfloat16))
    want = torch.full_like(wt, 7.0)
    for c in range(cols):
        at = off_t + c * ld
        want[:, at:at + rows] = w16[:, 8 + c:8 + rows * cols:cols]
    assert torch.equal(wt, want)


@pytest.mark.parametrize('m,n,with32', [(128, 64, True), (31, 33, True), (640, 649, True), (640, 649, False), (256, 96, False)])
def test_silu_derivative_bf16_output_is_the_rounded_f32(m, n, with32):
    """The bf16 result of the SiLU' epilogue over its range, NaN and infinities among it, is its f32
    result rounded, and the same without the f32 result (pairs of columns, whole and partial blocks)."""
    a = torch.ones(1, m, 8, dtype=torch.bfloat16, device='cuda') / 8
    b = torch.ones(1, n, 8, dtype=torch.bfloat16, device='cuda')
    z = torch.linspace(-100, 100, m * n).reshape(m, n)
    z[0, 0], z[0, 1], z[1, 0], z[1, 1] = float('nan'), float('inf'), float('-inf'), 0.0
    zc = z.cuda()
    out16, f32 = torch.zeros(2, m, n, dtype=torch.bfloat16, device='cuda'), torch.zeros(1, m, n, device='cuda')
    for i, keep in enumerate((True, with32)):
        more = dict(c2=f32.data_ptr(), ldc2=n, stride_c2=m * n) if keep else {}
        q = _problem(_abi.EPI_DSILU, m, n, 8, a, b, out16[i:i + 1], 0, 0, aux=zc.data_ptr(), ldaux=n, stride_aux=m * n, **more)
        assert _abi.load().mcw_mlp_gemm_batch(ctypes.byref(q), 1, _stream()) == 0
    torch.cuda.synchronize()
    want = f32[0].to(torch.bfloat16).float()
    assert torch.isnan(want[0, 0]) and torch.isfinite(want).sum() >= m * n - 3
    for i in range(2):
        assert torch.allclose(out16[i].float(), want, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize('G,B,rows,n_out', [(1, 1, 1, 1), (2, 33, 70, 649), (3, 64, 128, 40)])
def test_gather_and_grouped_loss(G, B, rows, n_out):
    """A step's batch with its transposed inputs, rows past the epoch's left alone, and the loss of
    grouped outputs with its gradient in f32, bf16 and bf16 transposed."""
    g = torch.Generator().manual_seed(B)
    x_all = torch.randn(rows, 16, generator=g).to(torch.bfloat16).cuda()
    t_all = torch.randn(rows, n_out, generator=g).cuda()
    perm = torch.stack([torch.randperm(rows, generator=g) for _ in range(G)]).int().cuda()
    L = _abi.load()
    last = (rows - 1) // B                                    # the epoch's last batch, cut short
    for c in (0, last):
        x, t = torch.full((G, B, 16), 7.0, dtype=torch.bfloat16, device='cuda'), torch.full((G, B, n_out), 7.0, device='cuda')
        xt = torch.full((G, 16, B), 7.0, dtype=torch.bfloat16, device='cuda')
        counter = torch.tensor([c], dtype=torch.int32, device='cuda')
        assert L.mcw_mlp_gather(x_all.data_ptr(), t_all.data_ptr(), n_out, n_out, perm.data_ptr(), rows, counter.data_ptr(),
                                B, G, x.data_ptr(), B * 16, xt.data_ptr(), 16 * B, t.data_ptr(), n_out, B * n_out,
                                _stream()) == 0
        torch.cuda.synchronize()
        for k in range(G):
            at = perm[k, c * B:(c + 1) * B].long()
            assert torch.equal(x[k, :at.numel()], x_all[at]) and torch.equal(t[k, :at.numel()], t_all[at])
            assert torch.equal(xt[k], x[k].t()) and (x[k, at.numel():] == 7).all() and (t[k, at.numel():] == 7).all()
    y, tt = torch.randn(G, B, n_out, generator=g).cuda(), torch.randn(G, B, n_out, generator=g).cuda()
    w = torch.rand(n_out, generator=g).cuda()
    g32, loss = torch.zeros(G, B, n_out, device='cuda'), torch.zeros(G, device='cuda')
    g16, g16t = torch.zeros(G, B, n_out, dtype=torch.bfloat16, device='cuda'), torch.zeros(G, n_out, B, dtype=torch.bfloat16, device='cuda')
    assert L.mcw_mlp_loss_grouped(y.data_ptr(), n_out, B * n_out, tt.data_ptr(), n_out, B * n_out, w.data_ptr(), G, B, n_out,
                                  g32.data_ptr(), n_out, B * n_out, g16.data_ptr(), B * n_out, g16t.data_ptr(), B, n_out * B,
                                  loss.data_ptr(), _stream()) == 0
    torch.cuda.synchronize()
    d = (y - tt).double()
    # (FP32 sums of at most 2e4 terms: 1e-5 of the whole; a gradient has four roundings)
    assert torch.allclose(loss.double(), (w.double() * d * d).mean((1, 2)), rtol=1e-5)
    assert torch.allclose(g32.double(), 2 * w.double() * d / (B * n_out), rtol=1e-6, atol=0)
    assert torch.equal(g16, g32.to(torch.bfloat16)) and torch.equal(g16t, g16.transpose(1, 2))


def test_empty_products_are_nothing():
    """A grouped product without rows or columns is nothing to do, whatever its operands' alignment and
    pitches, alone and among others of a launch."""
    a, b = torch.zeros(1, 128, 72, dtype=torch.bfloat16, device='cuda'), torch.ones(1, 64, 72, dtype=torch.bfloat16, device='cuda')
    c = torch.full((1, 128, 64), 7.0, device='cuda')
    for m, n, off, epi in ((0, 64, 0, _abi.EPI_F32), (128, 0, 2, _abi.EPI_F32), (0, 64, 2, _abi.EPI_BIAS_SILU)):
        p = _abi.GemmGroupedC(m, n, 72, 1, 1, epi, a.data_ptr() + off, 71, 0, b.data_ptr(), 72, 0, None, 0, None, 0, 0,
                              c.data_ptr(), 64, 0, 0, None, 0, 0, None, 0, 0)
        assert _abi.load().mcw_mlp_gemm_grouped(ctypes.byref(p), _stream()) == 0
    torch.cuda.synchronize()
    assert (c == 7).all()
    two = (_abi.GemmProblemC * 2)(_problem(_abi.EPI_LOSS, 0, 64, 72, a, b, c, 0, 0), _problem(_abi.EPI_F32, 128, 64, 72, a, b, c, 0, 0))
    assert _abi.load().mcw_mlp_gemm_batch(two, 2, _stream()) == 0
    torch.cuda.synchronize()
    assert (c == 0).all()
