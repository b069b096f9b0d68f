"""Threshold MLP: the CUDA forward/backward/Adam kernels against the float64 CPU oracle."""

import ctypes
import re
from pathlib import Path

import numpy as np
import pytest

from oracle import mlp_oracle as mo


def test_oracle_gradient_matches_central_differences():
    rng = np.random.default_rng(1)
    p = mo.init(3).astype(np.float64)
    x = rng.normal(size=(40, mo.IN))
    t = rng.normal(size=40)
    g = mo.gradient(p, x, t, 4.0)
    for q in rng.choice(mo.PARAMS, size=60, replace=False):
        h = 1e-6
        pp, pm = p.copy(), p.copy()
        pp[q] += h
        pm[q] -= h
        num = (mo.loss(pp, x, t, 4.0) - mo.loss(pm, x, t, 4.0)) / (2 * h)
        assert abs(num - g[q]) <= 1e-6 + 1e-4 * abs(num), (q, num, g[q])


def test_param_count_matches_oracle(pkg):
    assert pkg._native.engine_library().bm25_mlp_param_count() == mo.PARAMS


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.gpu
def test_forward_and_gradient_match_oracle(pkg, cuda_ok):
    import torch
    lib = pkg._native.engine_library()
    rng = np.random.default_rng(7)
    p = mo.init(11)
    batch = 300  # not a multiple of the kernels' row blocks
    x = rng.normal(size=(batch, mo.IN)).astype(np.float32)
    t = rng.normal(size=batch).astype(np.float32)
    dp, dx, dt = _dev(torch, p), _dev(torch, x), _dev(torch, t)
    y = torch.empty(batch, dtype=torch.float32, device='cuda')
    assert lib.bm25_mlp_forward(dp.data_ptr(), dx.data_ptr(), batch, y.data_ptr(), None) == 0
    ref = mo.forward(p, x)
    assert np.allclose(y.cpu().numpy(), ref, rtol=1e-5, atol=1e-5)
    scratch = torch.empty(lib.bm25_mlp_scratch_floats(batch), dtype=torch.float32, device='cuda')
    g = torch.empty(mo.PARAMS, dtype=torch.float32, device='cuda')
    loss = torch.empty(1, dtype=torch.float32, device='cuda')
    assert lib.bm25_mlp_gradient(dp.data_ptr(), dx.data_ptr(), dt.data_ptr(), batch, ctypes.c_float(4.0),
                                 scratch.data_ptr(), g.data_ptr(), loss.data_ptr(), None) == 0
    gref = mo.gradient(p, x, t, 4.0)
    gg = g.cpu().numpy()
    scale = np.abs(gref).max()
    assert np.abs(gg - gref).max() <= 1e-4 * scale, np.abs(gg - gref).max() / scale
    assert abs(loss.item() - mo.loss(p, x, t, 4.0)) <= 1e-4 * mo.loss(p, x, t, 4.0)
    # deterministic: the same call gives the same bits
    g2 = torch.empty_like(g)
    lib.bm25_mlp_gradient(dp.data_ptr(), dx.data_ptr(), dt.data_ptr(), batch, ctypes.c_float(4.0),
                          scratch.data_ptr(), g2.data_ptr(), None, None)
    assert torch.equal(g, g2)


@pytest.mark.gpu
def test_adam_training_fits_a_smooth_target(pkg, cuda_ok):
    import torch
    lib = pkg._native.engine_library()
    rng = np.random.default_rng(3)
    batch = 2048
    x = rng.normal(size=(batch, mo.IN)).astype(np.float32)
    t = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2] - 0.3 * np.abs(x[:, 3])).astype(np.float32)
    dp = _dev(torch, mo.init(5))
    m = torch.zeros(mo.PARAMS, device='cuda')
    v = torch.zeros(mo.PARAMS, device='cuda')
    dx, dt = _dev(torch, x), _dev(torch, t)
    scratch = torch.empty(lib.bm25_mlp_scratch_floats(batch), dtype=torch.float32, device='cuda')
    g = torch.empty(mo.PARAMS, device='cuda')
    loss = torch.empty(1, device='cuda')
    first = None
    for step in range(1, 301):
        assert lib.bm25_mlp_gradient(dp.data_ptr(), dx.data_ptr(), dt.data_ptr(), batch, ctypes.c_float(1.0),
                                     scratch.data_ptr(), g.data_ptr(), loss.data_ptr(), None) == 0
        if first is None:
            first = loss.item()
        assert lib.bm25_mlp_adam(dp.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), ctypes.c_float(3e-3), step,
                                 None) == 0
    torch.cuda.synchronize()
    final = mo.loss(dp.cpu().numpy(), x, t, 1.0)
    assert final < 0.2 * first, (first, final)


@pytest.mark.gpu
@pytest.mark.parametrize('batch', [1, 31, 32, 33, 1023, 1025, 4097])  # the row block, and 32 blocks' sums at a time
def test_gradient_at_row_block_edges(pkg, cuda_ok, batch):
    import torch
    lib = pkg._native.engine_library()
    rng = np.random.default_rng(batch)
    p = mo.init(5)
    x = rng.normal(size=(batch, mo.IN)).astype(np.float32)
    t = rng.normal(size=batch).astype(np.float32)
    dp, dx, dt = _dev(torch, p), _dev(torch, x), _dev(torch, t)
    scratch = torch.full((lib.bm25_mlp_scratch_floats(batch),), float('nan'), dtype=torch.float32, device='cuda')
    g = torch.empty(mo.PARAMS, dtype=torch.float32, device='cuda')
    loss = torch.empty(1, dtype=torch.float32, device='cuda')
    assert lib.bm25_mlp_gradient(dp.data_ptr(), dx.data_ptr(), dt.data_ptr(), batch, ctypes.c_float(4.0),
                                 scratch.data_ptr(), g.data_ptr(), loss.data_ptr(), None) == 0
    # FP32 chains of at most 64 + 32 + batch / 32 terms: 1e-4 of the largest entry covers their rounding
    gref = mo.gradient(p, x, t, 4.0)
    assert np.abs(g.cpu().numpy() - gref).max() <= 1e-4 * np.abs(gref).max()
    assert abs(loss.item() - mo.loss(p, x, t, 4.0)) <= 1e-4 * mo.loss(p, x, t, 4.0)


@pytest.mark.gpu
@pytest.mark.parametrize('batch', [1, 33, 1025])
def test_train_steps_are_gradient_and_adam_on_the_gathered_rows(pkg, cuda_ok, batch):
    import torch
    lib = pkg._native.engine_library()
    rng = np.random.default_rng(batch)
    x, t = _dev(torch, rng.normal(size=(2000, mo.IN))), _dev(torch, rng.normal(size=2000))
    rows = torch.from_numpy(rng.integers(0, 2000, (5, batch))).cuda()
    scratch = torch.empty(lib.bm25_mlp_scratch_floats(batch), dtype=torch.float32, device='cuda')
    want = [_dev(torch, mo.init(9)), torch.zeros(mo.PARAMS, device='cuda'), torch.zeros(mo.PARAMS, device='cuda')]
    got = [a.clone() for a in want]
    g, loss, losses = torch.empty(mo.PARAMS, device='cuda'), torch.empty(5, device='cuda'), torch.empty(5, device='cuda')
    for i in range(5):
        xb, tb = x[rows[i]].contiguous(), t[rows[i]].contiguous()
        assert lib.bm25_mlp_gradient(want[0].data_ptr(), xb.data_ptr(), tb.data_ptr(), batch, ctypes.c_float(4.0),
                                     scratch.data_ptr(), g.data_ptr(), loss[i:].data_ptr(), None) == 0
        assert lib.bm25_mlp_adam(want[0].data_ptr(), want[1].data_ptr(), want[2].data_ptr(), g.data_ptr(),
                                 ctypes.c_float(2e-3), i + 1, None) == 0
        torch.cuda.synchronize()
    for first in (0, 2):  # in two calls
        n = 2 if first == 0 else 3
        assert lib.bm25_mlp_train_steps(got[0].data_ptr(), got[1].data_ptr(), got[2].data_ptr(), x.data_ptr(),
                                        t.data_ptr(), rows[first:].data_ptr(), batch, n, first + 1, 4.0, 2e-3,
                                        scratch.data_ptr(), losses[first:].data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got + [losses], want + [loss]))


def test_overlapped_backward_makes_no_promise_of_constant_parameters():
    """A training step's backward kernel starts while the update before it writes the parameters: a
    __restrict__ const argument or a read-only load of them may be moved above the wait."""
    src = (Path(__file__).resolve().parents[1] / 'bm25-npu_b200' / 'csrc' / 'mlp.cu').read_text()
    kernel = re.search(r'BackwardKernel\(const float \*.*?\n}\n', src, re.S).group()
    signature, body = kernel.split('{', 1)
    assert re.match(r'BackwardKernel\(const float \*p,', signature), signature
    before, after = body.split('WaitPrerequisites();')
    assert not re.search(r'\bp\b', before)  # nothing of p is read before the wait
    assert not re.search(r'\bp\[|__ldg\(p\b', after) and after.count('__ldcg(p + ') == 6


@pytest.mark.gpu
@pytest.mark.parametrize('batch', [4096, 4097])  # 128 and 129 CTAs: the backward kernel on nearly every SM
def test_overlapped_training_steps_see_each_update(pkg, cuda_ok, batch):
    """Twelve overlapped steps in one call have the bits of separate gradient and Adam calls."""
    import torch
    lib = pkg._native.engine_library()
    steps = 12
    rng = np.random.default_rng(batch)
    x, t = _dev(torch, rng.normal(size=(9000, mo.IN))), _dev(torch, rng.normal(size=9000))
    rows = torch.from_numpy(rng.integers(0, 9000, (steps, batch))).cuda()
    scratch = torch.empty(lib.bm25_mlp_scratch_floats(batch), dtype=torch.float32, device='cuda')
    want = [_dev(torch, mo.init(9)), torch.zeros(mo.PARAMS, device='cuda'), torch.zeros(mo.PARAMS, device='cuda')]
    got = [a.clone() for a in want]
    g = torch.empty(mo.PARAMS, device='cuda')
    loss, losses = torch.empty(steps, device='cuda'), torch.empty(steps, device='cuda')
    for i in range(steps):
        xb, tb = x[rows[i]].contiguous(), t[rows[i]].contiguous()
        torch.cuda.synchronize()
        assert lib.bm25_mlp_gradient(want[0].data_ptr(), xb.data_ptr(), tb.data_ptr(), batch, ctypes.c_float(4.0),
                                     scratch.data_ptr(), g.data_ptr(), loss[i:].data_ptr(), None) == 0
        assert lib.bm25_mlp_adam(want[0].data_ptr(), want[1].data_ptr(), want[2].data_ptr(), g.data_ptr(),
                                 ctypes.c_float(2e-3), i + 1, None) == 0
        torch.cuda.synchronize()
    assert lib.bm25_mlp_train_steps(got[0].data_ptr(), got[1].data_ptr(), got[2].data_ptr(), x.data_ptr(),
                                    t.data_ptr(), rows.data_ptr(), batch, steps, 1, 4.0, 2e-3, scratch.data_ptr(),
                                    losses.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got + [losses], want + [loss]))


@pytest.mark.parametrize('features,targets', [((50, 31), (50,)), ((50, 33), (50,)), ((50, 32), (49,)),
                                              ((50, 32), (50, 2)), ((64,), (64,))])
def test_train_refuses_features_the_kernel_would_misread(pkg, features, targets):
    """Rows of another width than 32, or fewer targets than rows, are refused before the device is used."""
    with pytest.raises(ValueError, match='features'):
        pkg.learned.train(np.zeros(features, np.float32), np.zeros(targets, np.float32), steps=1)


@pytest.mark.gpu
@pytest.mark.parametrize('features,targets', [((40, 32), (40,)), ((40, 32), (40, 1)), ((40, 4, 8), (40,)),
                                              ((40, 32), (45,))])
def test_train_accepts_whole_rows(pkg, cuda_ok, features, targets):
    """Any shape that holds 32 features and one target per row trains the same model."""
    rng = np.random.default_rng(1)
    x, t = rng.normal(size=(40, 32)).astype(np.float32), rng.normal(size=40).astype(np.float32)
    want, want_loss = pkg.learned.train(x, t, steps=9, batch=16)
    y = np.full(int(np.prod(targets)), t.mean(), np.float32)
    y[:40] = t
    got, loss = pkg.learned.train(x.reshape(features), y.reshape(targets), steps=9, batch=16)
    if y.size == 40:
        assert np.array_equal(got, want) and np.array_equal(loss, want_loss)
    else:  # the targets' mean starts the bias: equal to rounding
        assert np.allclose(got, want, atol=1e-4) and np.allclose(loss, want_loss, rtol=1e-3)
