"""What Net.load takes and refuses: the arrays it is given fill rows x T_IN x 2 and rows x AUX, are broadcast
to them as a tensor assignment does, or are refused; no launch reads more values than an array holds. The
kernel that lays them out is replaced by a copy on the host, so no device is needed."""
import ctypes as C

import numpy as np
import pytest
import torch

from em_lab_gb300 import extrap
from em_lab_gb300.extrap import AUX, ENC, OUT, T_IN

BATCH = 6


class HostKernels:
    """emlab_nn_pad_to_bf16 and emlab_nn_to_bf16 on host memory; refuses to read past a tracked array."""

    def __init__(self):
        self.sizes = {}

    def emlab_nn_to_bf16(self, *a):
        return 0

    def emlab_nn_pad_to_bf16(self, src, given, n, out, ldo, cols, off, stream):
        assert given <= self.sizes.get(src, given), "reads past its input"
        x = np.zeros(n, np.float32)
        if given:
            x[:given] = np.frombuffer(C.string_at(src, given * 4), np.float32)
        rows = n // cols
        bits = torch.from_numpy(x.reshape(rows, cols)).bfloat16().view(torch.int16).numpy()
        for r in range(rows):
            C.memmove(out + 2 * (r * ldo + off), np.ascontiguousarray(bits[r]).ctypes.data, 2 * cols)
        return 0


@pytest.fixture
def net(monkeypatch):
    lib = HostKernels()
    monkeypatch.setattr(extrap, "_nn_lib", lambda: lib)
    monkeypatch.setattr(extrap.Net, "stream", property(lambda self: None))
    n = extrap.Net(extrap.init_params(3), BATCH, "cpu")
    real = torch.from_numpy

    def tracked(a):
        t = real(a)
        lib.sizes[t.data_ptr()] = t.numel()
        return t

    monkeypatch.setattr(torch, "from_numpy", tracked)
    return n


def loaded(net):
    return net.x0.float().numpy(), net.X0.float().numpy()[:, ENC:]


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).bfloat16().float().numpy()


@pytest.mark.parametrize("n", [1, 4, BATCH])
@pytest.mark.parametrize("shape", [(AUX,), (1, AUX), (), (1, 1), (None, 1), (None, AUX), (1, None, AUX)])
def test_head_inputs_are_broadcast_to_the_rows(net, n, shape):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, T_IN, 2)).astype(np.float32)
    zt = rng.standard_normal([n if s is None else s for s in shape]).astype(np.float32)
    net.load(x, zt)
    got_x, got_z = loaded(net)
    np.testing.assert_array_equal(got_x[:n], bf16(x))
    np.testing.assert_array_equal(got_z[:n], np.broadcast_to(bf16(zt), (1, n, AUX))[0])
    assert not got_x[n:].any() and not got_z[n:].any() and net.n == n


@pytest.mark.parametrize("shape", [(4, T_IN, 1), (4, 1, 2), (4, 1, 1)])
def test_inputs_are_broadcast_to_the_samples(net, shape):
    x = np.random.default_rng(1).standard_normal(shape)
    net.load(x, np.zeros((4, AUX)))
    np.testing.assert_array_equal(loaded(net)[0][:4], np.broadcast_to(bf16(x), (4, T_IN, 2)))


@pytest.mark.parametrize("xs,zs,ts", [((4, T_IN, 2), (3, AUX), None), ((4, T_IN, 2), (5, AUX), None),
                                      ((4, T_IN, 2), (4, AUX - 1), None), ((4, T_IN, 2), (4, AUX + 1), None),
                                      ((4, T_IN - 1, 2), (4, AUX), None), ((4, T_IN + 1, 2), (4, AUX), None),
                                      ((4, T_IN, 3), (4, AUX), None), ((4, 2 * T_IN), (4, AUX), None),
                                      ((4, T_IN, 2), (4, AUX), (3, OUT)), ((4, T_IN, 2), (4, AUX), (4, OUT - 1))])
def test_other_shapes_are_refused(net, xs, zs, ts):
    with pytest.raises(RuntimeError):
        net.load(np.zeros(xs), np.zeros(zs), None if ts is None else np.zeros(ts))


def test_predict_refuses_fewer_head_rows_than_samples(net):
    with pytest.raises(RuntimeError):
        net.predict(np.zeros((4, T_IN, 2)), np.zeros((2, AUX)))


def test_targets_are_broadcast_to_the_rows(net):
    t = np.random.default_rng(2).standard_normal((1, 1, OUT))
    net.load(np.zeros((4, T_IN, 2)), np.zeros((4, AUX)), t)
    np.testing.assert_array_equal(net.t[:4].numpy(), np.broadcast_to(t.astype(np.float32)[0], (4, OUT)))
