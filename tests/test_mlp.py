"""Radiance-cache tensor-core kernels: operand layouts (GEMM self-test),
network forward/backward against an fp64 CPU restatement, training."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def to_bf16(x):
    u = np.ascontiguousarray(x, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) >> 16
    return u.astype(np.uint16)


def from_bf16(b):
    return (b.astype(np.uint32) << 16).view(np.float32)


@pytest.mark.parametrize("mode,K,N", [(0, 16, 16), (0, 64, 64), (0, 80, 64), (0, 64, 16), (0, 128, 32),
                                      (1, 64, 64), (1, 80, 64), (1, 64, 16), (1, 128, 16),
                                      (2, 16, 64), (2, 64, 64), (2, 128, 32)])
def test_umma_gemm_layouts(vrt, mode, K, N):
    import ctypes as C
    rng = np.random.default_rng(K * 7 + N + mode)
    A = to_bf16(rng.normal(size=(128, K)))
    B = to_bf16(rng.normal(size={0: (N, K), 1: (128, N), 2: (K, N)}[mode]))
    D = np.zeros((128, N), np.float32)
    code = vrt.lib.vrt_mlp_selftest_gemm(mode, K, N, C.c_void_p(A.ctypes.data), C.c_void_p(B.ctypes.data),
                                         C.c_void_p(D.ctypes.data))
    assert code == 0, vrt.lib.vrt_last_error_string().decode()
    a, b = from_bf16(A).astype(np.float64), from_bf16(B).astype(np.float64)
    ref = {0: lambda: a @ b.T, 1: lambda: a.T @ b, 2: lambda: a @ b}[mode]()
    rows = K if mode == 1 else 128
    err = np.abs(D[:rows] - ref) / (np.abs(ref) + 1.0)
    assert err.max() < 1e-5, f"max err {err.max()}"


EXTENT = 16.0


def _queries(rng, n, extent=EXTENT):
    q = np.zeros((n, 9), np.float32)
    q[:, :3] = rng.uniform(-0.25 * extent, 1.25 * extent, size=(n, 3))   # outside the world too
    nrm = rng.normal(size=(n, 3))
    q[:, 3:6] = nrm / np.linalg.norm(nrm, axis=1, keepdims=True)
    q[:, 6:9] = rng.uniform(0, 1, size=(n, 3))
    y = (q[:, 6:9] * (0.6 + 0.4 * np.sin(q[:, :1] * 0.9) * np.cos(q[:, 2:3] * 0.5)) *
         (1.0 + q[:, 4:5])).astype(np.float32)
    return q, y


def _cuda(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture
def cache(vrt):
    ctx = vrt.Context(0)
    rc = vrt.RadianceCache(ctx, seed=7, extent=EXTENT)
    yield rc
    rc.close()
    ctx.close()


@pytest.mark.parametrize("n", [1, 127, 1000])
def test_mlp_encode_bit_exact(vrt, orc, cache, n):
    import torch
    from oracle import mlp_ref as M
    q, _ = _queries(np.random.default_rng(n), n)
    feat = torch.zeros(n * 80, dtype=torch.int16, device="cuda")
    cache.encode(_cuda(q), feat)
    got = feat.cpu().numpy().view(np.uint16).reshape(n, 80)
    want = M.bf16_bits(M.encode(q, EXTENT))
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n", [1, 200, 5000])
def test_mlp_infer_matches_oracle(vrt, orc, cache, n):
    import torch
    from oracle import mlp_ref as M
    q, _ = _queries(np.random.default_rng(10 + n), n)
    out = torch.zeros(n * 3, dtype=torch.float32, device="cuda")
    cache.infer(_cuda(q), out)
    got = out.cpu().numpy().reshape(n, 3)
    o, _, _ = M.forward(M.encode(q, EXTENT), cache.params())
    ref = o[:, :3]
    # fp32 tensor-core sums vs fp64 sums: outputs agree to 1e-5 of the output
    # scale except where a hidden activation sits on a bf16 rounding boundary
    # and rounds the other way (a relative step of 2^-8 in one activation):
    # at most 1% of the outputs, each within 5e-3 of the scale
    scale = max(np.abs(ref).max(), 1e-3)
    err = np.abs(got - ref)
    assert err.max() <= 5e-3 * scale, err.max()
    assert np.mean(err > 1e-5 * scale) <= 0.01, np.mean(err > 1e-5 * scale)


@pytest.mark.parametrize("n", [1, 3000, 148 * 128 * 2 + 77])
def test_mlp_gradient_matches_oracle(vrt, orc, cache, n):
    """Backward pass (dX by K-major MMAs, dW by MN-major MMAs accumulated in
    TMEM over a CTA's tiles, fixed-order cross-CTA reduction) against the
    restatement; the largest case gives every CTA two or three tiles."""
    import torch
    from oracle import mlp_ref as M
    rng = np.random.default_rng(20 + n)
    q, y = _queries(rng, n)
    p = cache.params()
    g = torch.zeros(M.N_PARAMS, dtype=torch.float32, device="cuda")
    loss = cache.gradient(_cuda(q), _cuda(y), g)
    got = g.cpu().numpy()
    want_loss, want = M.gradient(M.encode(q, EXTENT), y, p)
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss) + 1e-7, (loss, want_loss)
    # per layer: |gpu - oracle| <= 2e-3 * max|oracle| + 1e-2 * |oracle|; the
    # relative Frobenius error stays below 2e-3
    off = 0
    for k, m in M.SHAPES:
        a, b = got[off:off + k * m], want[off:off + k * m]
        scale = np.abs(b).max()
        assert np.all(np.abs(a - b) <= 2e-3 * scale + 1e-2 * np.abs(b)), (k, m, np.abs(a - b).max(), scale)
        off += k * m
    assert np.linalg.norm(got - want) <= 2e-3 * np.linalg.norm(want)


def test_mlp_gradient_deterministic(vrt, cache):
    import torch
    q, y = _queries(np.random.default_rng(5), 40000)
    qd, yd = _cuda(q), _cuda(y)
    g1 = torch.zeros(14336, dtype=torch.float32, device="cuda")
    g2 = torch.zeros_like(g1)
    l1 = cache.gradient(qd, yd, g1)
    l2 = cache.gradient(qd, yd, g2)
    assert l1 == l2
    assert torch.equal(g1, g2)


def test_mlp_adam_step_matches_oracle(vrt, orc, cache):
    import torch
    from oracle import mlp_ref as M
    q, y = _queries(np.random.default_rng(6), 4096)
    qd, yd = _cuda(q), _cuda(y)
    w0 = cache.params()
    cache.set_params(w0)                      # zero Adam state
    m = np.zeros_like(w0)
    v = np.zeros_like(w0)
    w = w0
    g = torch.zeros(M.N_PARAMS, dtype=torch.float32, device="cuda")
    for step in (1, 2, 3):
        cache.gradient(qd, yd, g)             # the gradient the next step uses
        cache.train(qd, yd, lr=1e-3, steps=1)
        w, m, v = M.adam(w, m, v, g.cpu().numpy(), step, 1e-3)
        np.testing.assert_allclose(cache.params(), w, rtol=1e-5, atol=1e-7)


def test_mlp_training_reduces_loss(vrt, cache):
    q, y = _queries(np.random.default_rng(7), 16384)
    qd, yd = _cuda(q), _cuda(y)
    l0 = cache.train(qd, yd, lr=1e-2, steps=1)
    for _ in range(6):
        cache.train(qd, yd, lr=1e-2, steps=50)
    l1 = cache.gradient(qd, yd)
    assert np.isfinite(l1) and l1 < 0.2 * l0, (l0, l1)


def test_mlp_rejects_bad_arguments(vrt, cache):
    import torch
    q = torch.zeros(9, dtype=torch.float32, device="cuda")
    y = torch.zeros(3, dtype=torch.float32, device="cuda")
    from voxelrt_b200._lib import lib
    import ctypes as C
    assert lib.vrt_mlp_train_device(cache.h, C.c_void_p(q.data_ptr()), C.c_void_p(y.data_ptr()), 0,
                                    C.c_float(16.0), C.c_float(1e-3), 1, None) != 0
    assert lib.vrt_mlp_infer_device(cache.h, C.c_void_p(q.data_ptr()), 1, C.c_float(0.0), C.c_void_p(y.data_ptr())) != 0


def test_bounded_wait_runs_out_and_context_survives(vrt, cache):
    """A wait that nothing completes gives up after its bound, reports
    VRT_ERR_TIMEOUT through the status code, frees its TMEM, and the device
    keeps working (an inference afterwards succeeds)."""
    import torch
    from voxelrt_b200._lib import lib
    assert lib.vrt_selftest_bounded_wait(1000) == 6        # VRT_ERR_TIMEOUT
    assert b"ran out" in lib.vrt_last_error_string()
    q, _ = _queries(np.random.default_rng(9), 300)
    out = torch.zeros(900, dtype=torch.float32, device="cuda")
    cache.infer(_cuda(q), out)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("tiny", [1e-20, 1e-23])
def test_gradient_through_tiny_activations(vrt, orc, cache, tiny):
    """A positive pre-activation below half of bf16's least value (tiny * 1e-21) is stored as next to nothing, but the
    ReLU's derivative there is 1.  Tolerance: that of test_mlp_gradient_matches_oracle."""
    import torch
    from oracle import mlp_ref as M
    rng = np.random.default_rng(3)
    q, y = _queries(rng, 700)
    ws = [rng.normal(size=s).astype(np.float32) * np.float32(0.1) for s in M.SHAPES]
    ws[3][:, 3:] = 0.0
    ws[0][:, 3] = 0.0
    ws[0][78, 3] = tiny                        # feature 78 is the constant 1
    ws[1][:, 7] = 0.0
    ws[1][3, 7] = 1e-21
    ws[2][7, :] = 1.0
    p = M.pack(ws).astype(np.float32)
    cache.set_params(p)
    g = torch.zeros(M.N_PARAMS, dtype=torch.float32, device="cuda")
    cache.gradient(_cuda(q), _cuda(y), g)
    got, want = M.unpack(g.cpu().numpy())[1], M.unpack(M.gradient(M.encode(q, EXTENT), y, p)[1])[1]
    assert np.abs(want[:, 7]).max() > 0.1 * np.abs(want).max()
    assert np.all(np.abs(got - want) <= 2e-3 * np.abs(want).max() + 1e-2 * np.abs(want))


def test_gradient_with_a_nan_query(vrt, cache):
    """The pre-activations of a NaN query are NaN and count as 0: its sample adds to the loss and to no gradient but
    that of the weights its NaN feature meets.  So the sum over 257 samples with it is the sum over the 256 without it
    (both means carry two fp32 roundings)."""
    import torch
    q, y = _queries(np.random.default_rng(4), 257)
    q[256, 3] = np.nan                          # feature 72
    out = []
    for n in (256, 257):
        g = torch.zeros(14336, dtype=torch.float32, device="cuda")
        loss = cache.gradient(_cuda(q[:n]), _cuda(y[:n]), g)
        assert np.isfinite(loss)
        out.append(g.cpu().numpy().astype(np.float64) * n)
    keep = np.ones(14336, bool)
    keep[72 * 64:73 * 64] = False
    np.testing.assert_allclose(out[1][keep], out[0][keep], rtol=4 * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("shift", [0, 4, 6])
def test_gradient_into_any_alignment(vrt, cache, shift):
    """The caller's array at byte offsets that a kernel can (0, 4) and cannot (6) store floats to."""
    import ctypes as C

    import torch
    q, y = (_cuda(a) for a in _queries(np.random.default_rng(6), 300))
    want = torch.zeros(14336, dtype=torch.float32, device="cuda")
    loss = cache.gradient(q, y, want)
    buf = torch.full((14336 * 4 + 16,), 0x55, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for with_loss in (True, False):
        got = C.c_float()
        code = vrt.lib.vrt_mlp_gradient_device(cache.h, C.c_void_p(q.data_ptr()), C.c_void_p(y.data_ptr()), 300,
                                               C.c_float(EXTENT), C.c_void_p(buf.data_ptr() + shift),
                                               C.byref(got) if with_loss else None)
        assert code == 0, vrt.lib.vrt_last_error_string().decode()
        b = buf.cpu().numpy()
        assert b[shift:shift + 14336 * 4].tobytes() == want.cpu().numpy().tobytes()
        assert np.all(b[:shift] == 0x55) and np.all(b[shift + 14336 * 4:] == 0x55)
        assert not with_loss or got.value == loss
