"""GEMMs with the bias, activation and gradient steps in their epilogue, and the weight gradients whose ring
holds several chunks a round, against the separate entry points on the same inputs: equal bit for bit (the
same operations element by element, the same order of every sum), at sizes on both sides of the tiles, the
vector width and the chunk, with outputs that interleave rows and with part of the columns."""
import numpy as np
import pytest

from em_lab_gb300 import extrap
from em_lab_gb300.grid import _check

pytestmark = pytest.mark.gpu


def _setup(seed):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    return torch, extrap._nn_lib(), rand, torch.cuda.current_stream().cuda_stream


def _fp(t):
    import ctypes as C
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_float))


@pytest.mark.parametrize("M,N,K,group", [(1, 1, 1, 1), (7, 33, 16, 1), (128, 64, 64, 4), (300, 40, 72, 3), (256, 256, 1344, 1),
                                         (4096, 64, 256, 16), (16384, 320, 64, 1)])
@pytest.mark.parametrize("relu,bias", [(1, True), (0, False)])
def test_bias_and_activation(M, N, K, group, relu, bias):
    torch, lib, rand, s = _setup(M + N)
    A, B, b = rand(M, K).bfloat16(), rand(N, K).bfloat16(), rand(N)
    ldo, off = group * N + 8, 8
    rows = -(-M // group)
    z, z0 = torch.zeros(M, N, device="cuda"), torch.zeros(M, N, device="cuda")
    out, out0 = torch.zeros(rows, ldo, device="cuda").bfloat16(), torch.zeros(M, N, device="cuda").bfloat16()
    _check(lib.emlab_nn_gemm_bias_act(M, N, K, A.data_ptr(), K, 1, B.data_ptr(), K, 1, z.data_ptr(), N,
                                      b.data_ptr() if bias else None, relu, out.data_ptr(), ldo, off, group, s))
    _check(lib.emlab_nn_gemm(M, N, K, A.data_ptr(), K, 1, B.data_ptr(), K, 1, _fp(z0), N, s))
    _check(lib.emlab_nn_bias_act(_fp(z0), _fp(b) if bias else None, M, N, N, relu, out0.data_ptr(), N, 0, s))
    assert torch.equal(z, z0)
    want = torch.zeros(rows * group, N, device="cuda").bfloat16()
    want[:M] = out0
    assert torch.equal(out[:, off:], want.reshape(rows, group * N)) and not out[:, :off].any()


@pytest.mark.parametrize("M,N,K,cols", [(1, 1, 1, 1), (7, 33, 16, 20), (130, 64, 64, 64), (64, 72, 40, 41), (256, 1344, 256, 1024)])
@pytest.mark.parametrize("relu", [0, 1])
def test_gradient_through_the_activation(M, N, K, cols, relu):
    torch, lib, rand, s = _setup(M + N + relu)
    A, B, z = rand(M, K).bfloat16(), rand(K, N).bfloat16(), rand(M, cols)
    z[0, 0] = 0.0
    dz, dz0 = torch.zeros(M, cols, device="cuda"), torch.zeros(M, cols, device="cuda")
    db, db0, dy = dz.bfloat16(), dz.bfloat16(), torch.zeros(M, N, device="cuda")
    _check(lib.emlab_nn_gemm_act_grad(M, N, K, A.data_ptr(), K, 1, B.data_ptr(), 1, N, z.data_ptr(), cols, relu,
                                      dz.data_ptr(), db.data_ptr(), s))
    _check(lib.emlab_nn_gemm(M, N, K, A.data_ptr(), K, 1, B.data_ptr(), 1, N, _fp(dy), N, s))
    _check(lib.emlab_nn_act_grad(_fp(dy), N, 0, _fp(z), M, cols, relu, _fp(dz0), db0.data_ptr(), s))
    assert torch.equal(dz, dz0) and torch.equal(db, db0)


@pytest.mark.parametrize("M,N,K", [(8, 8, 1), (32, 16, 16384), (64, 256, 4096), (64, 72, 63), (40, 24, 1000), (56, 200, 449),
                                   (72, 16, 300), (136, 64, 128)])
def test_weight_gradients_of_few_rows(M, N, K):
    torch, lib, rand, s = _setup(M + N + K)
    dz, x = rand(K, M), rand(K, N).bfloat16()
    db = dz.bfloat16()
    gw, gb, gw0, gb0 = (torch.full(sh, 7.0, device="cuda") for sh in ((M, N), (M,), (M, N), (M,)))
    g = (extrap._Grad * 1)()
    g[0].out_features, g[0].in_features, g[0].rows = M, N, K
    g[0].dz_bf16, g[0].x_bf16, g[0].dz, g[0].gw, g[0].gb = (t.data_ptr() for t in (db, x, dz, gw, gb))
    _check(lib.emlab_nn_weight_grads(g, 1, s))
    _check(lib.emlab_nn_gemm(M, N, K, db.data_ptr(), 1, M, x.data_ptr(), 1, N, _fp(gw0), N, s))
    _check(lib.emlab_nn_col_sum(_fp(dz), K, M, _fp(gb0), s))
    _check(lib.emlab_nn_status(s))
    assert torch.equal(gw, gw0) and torch.equal(gb, gb0)


@pytest.mark.parametrize("rows,batch", [(1, 32), (31, 32), (32, 32)])
def test_padded_rows_are_zero(rows, batch):
    torch, lib, rand, s = _setup(rows)
    y, t = rand(batch, 10), rand(batch, 10)
    dy, loss, loss0 = torch.full((batch, 10), 3.0, device="cuda"), torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    db, dy0 = dy.bfloat16(), torch.zeros(batch, 10, device="cuda")
    _check(lib.emlab_nn_mse_grad(y.data_ptr(), t.data_ptr(), rows * 10, batch * 10, dy.data_ptr(), db.data_ptr(),
                                 loss.data_ptr(), s))
    _check(lib.emlab_nn_mse(_fp(y), _fp(t), rows * 10, _fp(dy0), _fp(loss0), s))
    assert torch.equal(dy, dy0) and torch.equal(db, dy0.bfloat16())
    assert float(loss) == pytest.approx(float(loss0), rel=1e-6)
    out = torch.full((batch, 24), 5.0, device="cuda").bfloat16()
    _check(lib.emlab_nn_pad_to_bf16(y.data_ptr(), rows * 10, batch * 10, out.data_ptr(), 24, 10, 8, s))
    assert torch.equal(out[:rows, 8:18], y[:rows].bfloat16()) and not out[rows:, 8:18].any()
    assert np.all(out[:, :8].float().cpu().numpy() == 5.0)
