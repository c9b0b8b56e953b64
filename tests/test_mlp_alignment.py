"""Layer outputs whose base is not 16-byte aligned, at a row stride that 16-byte accesses could take: the same bits as
at an aligned base."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(64, 64), (128, 512), (256, 4096)])  # one and several splits of K
@pytest.mark.parametrize("shift", [1, 2, 4])
def test_shifted_bases(N, K, shift):
    torch = pytest.importorskip("torch")
    from symboltz import _lib
    L = _lib.lib()
    M, ldo = 128, N + 8
    g = torch.Generator(device="cuda").manual_seed(N + K)
    A = torch.randint(-3, 4, (M, K), device="cuda", generator=g).to(torch.bfloat16)  # integers: sums are exact in any order
    B = torch.randint(-3, 4, (N, K), device="cuda", generator=g).to(torch.bfloat16)
    z = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    res = []
    for sh in (0, shift):
        def at(dtype, fill):
            buf = torch.full((M * ldo + 16,), fill, device="cuda", dtype=dtype)
            return buf, buf[sh:sh + M * ldo].view(M, ldo), C.c_void_p(buf.data_ptr() + sh * buf.element_size())
        f, fv, fp = at(torch.float32, -5.0)
        y, yv, yp = at(torch.bfloat16, -5.0)
        d, dv, dp = at(torch.bfloat16, -5.0)
        zi, ziv, zip_ = at(torch.bfloat16, 0.0)
        zo, zov, zop = at(torch.bfloat16, -5.0)
        ziv[:, :N] = z
        a, b = C.c_void_p(A.data_ptr()), C.c_void_p(B.data_ptr())
        assert L.sbz_mlp_gemm(M, N, K, a, b, 0, 0, None, fp, ldo, 0, 0, None, None, st) == 0
        assert L.sbz_mlp_gemm(M, N, K, a, b, 1, 1, None, yp, ldo, 0, 0, zop, None, st) == 0
        assert L.sbz_mlp_gemm(M, N, K, a, b, 2, 1, None, dp, ldo, 0, 0, None, zip_, st) == 0
        for t in (fv, yv, dv, zov):
            assert (t[:, N:] == -5.0).all()
        res.append([t[:, :N].clone() for t in (fv, yv, dv, zov)])
    torch.testing.assert_close(res[0][0], A.float() @ B.float().T, rtol=0, atol=0)
    for p, q in zip(*res):
        assert torch.equal(p, q)
