"""Edges of the surrogate's tensor-core layers: the epilogue that stores through shared memory against the one
that stores from registers (the same product and the same roundings, so the same bits), and a training step on
ragged sizes against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N picks the tile (256, 128 or 64 columns; only the first two have the shared-memory route), K = 64 is one
# pipeline step; the last three have several tiles per CTA
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (384, 256, 192), (128, 384, 128), (256, 512, 64), (128, 640, 320), (128, 192, 64),
                                   (41216, 256, 64), (41216, 128, 192), (41088, 256, 128)])
@pytest.mark.parametrize("act", [0, 1])
def test_shared_memory_epilogue_has_the_register_epilogue_s_bits(M, N, K, act):
    torch = pytest.importorskip("torch")
    from symboltz import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = (0.2 * torch.randn(M, K, device="cuda", generator=g)).to(torch.bfloat16)
    B = (0.2 * torch.randn(N, K, device="cuda", generator=g)).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g)
    zin = (3 * torch.randn(M, N, device="cuda", generator=g)).to(torch.bfloat16)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    res = {}
    for ldo in (N + 8, N + 4):  # 16-byte row strides, and a stride that only the register route takes
        pad = lambda: torch.full((M, ldo), -7.0, device="cuda", dtype=torch.bfloat16)  # noqa: E731
        y, z, y2, dy, zi = pad(), pad(), pad(), pad(), pad()
        zi[:, :N] = zin
        assert L.sbz_mlp_gemm(M, N, K, p(A), p(B), 1, act, p(bias), p(y), ldo, 0, 0, p(z), None, st) == 0
        assert L.sbz_mlp_gemm(M, N, K, p(A), p(B), 1, act, None, p(y2), ldo, 0, 0, None, None, st) == 0
        assert L.sbz_mlp_gemm(M, N, K, p(A), p(B), 2, act, None, p(dy), ldo, 0, 0, None, p(zi), st) == 0
        for t in (y, z, y2, dy):
            assert (t[:, N:] == -7.0).all()  # nothing beyond the columns
        res[ldo] = [t[:, :N].clone() for t in (y, z, y2, dy)]
    for a, b in zip(res[N + 8], res[N + 4]):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    # half a bf16 ulp (2^-9) of z itself, and FP32 sums of K products of about 0.04
    ref = A.float() @ B.float().T + bias
    torch.testing.assert_close(res[N + 8][1].float(), ref, rtol=2.0 ** -8, atol=1e-5 * K)


# split K: partial tiles added by TMA (16-byte output rows) or by atomics (ldo = N + 2), in every tile width
@pytest.mark.parametrize("M,N,K", [(128, 64, 512), (128, 128, 4096), (256, 256, 8192), (128, 192, 2048)])
@pytest.mark.parametrize("pad", [0, 4, 2])
def test_split_k_sums(M, N, K, pad):
    torch = pytest.importorskip("torch")
    from symboltz import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    ref = A.double() @ B.double().T
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    out = torch.full((M, N + pad), 3.0, device="cuda")
    for acc in (0, 1):
        assert L.sbz_mlp_gemm(M, N, K, p(A), p(B), 0, 0, None, p(out), N + pad, 0, acc, None, None, st) == 0
        # FP32 sums of K products of order 1: K^(1/2) terms of one rounding (2^-24 of a partial sum of K^(1/2)) and margin
        torch.testing.assert_close(out[:, :N].double(), (1 + acc) * ref, rtol=0, atol=1e-6 * K * (1 + acc))
        assert (out[:, N:] == 3.0).all()


# widths of both tile sizes, odd input and output counts, batches of one and several row tiles; the gradient
# batch is smaller than the training batch (other strides in the same buffers), and comes after training steps
# (weights and their transposed copies as the optimiser left them)
@pytest.mark.parametrize("nin,width,nhidden,nout,batch,n", [(1, 128, 1, 1, 128, 128), (33, 256, 2, 5, 384, 128), (64, 384, 3, 64, 256, 256)])
def test_training_and_gradients_on_ragged_sizes(nin, width, nhidden, nout, batch, n):
    import mlp as MO
    from symboltz.surrogate import MLP
    net = MLP(nin, width, nhidden, nout, batch, 3)
    layers = MO.layer_sizes(nin, width, nhidden, nout)
    rng = np.random.default_rng(nin)
    X = rng.uniform(-1, 1, (n, nin)).astype(np.float32)
    Y = rng.normal(size=(n, nout)).astype(np.float32)
    # one data row: every batch row is that row, whatever the draw, so the loss is known
    net.set_data(X[:1], Y[:1])
    lo, _ = MO.loss_and_grad(net.get_params().astype(np.float64), X[:1], Y[:1], layers, bf16_operands=True)
    assert abs(net.train(1, 1e-3) - lo) <= 1e-2 * lo
    net.set_data(X, Y)
    net.train(3, 1e-3)
    p = net.get_params().astype(np.float64)
    loss, g = net.gradients(X, Y)
    lo, go = MO.loss_and_grad(p, X, Y, layers, bf16_operands=True)
    assert abs(loss - lo) <= 1e-2 * lo
    o = 0
    for a, b in zip(layers[:-1], layers[1:]):
        for m in (a * b, b):
            assert np.linalg.norm(g[o:o + m] - go[o:o + m]) <= 3e-2 * np.linalg.norm(go[o:o + m]), (a, b, m)
            o += m
    assert o == len(g)
