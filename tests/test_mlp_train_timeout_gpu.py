"""A training step whose bounded wait ran out (its status word set here from the host) leaves parameters and moments as
they were and is reported; without it the same step changes them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_update_after_a_timeout(gpu, tmp_path):
    import torch
    from cube2_b200 import build as B
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import CubeError
    so = str(tmp_path / "libmlp_probe.so")
    subprocess.run([B.NVCC, *B.ARCH, *B.FLAGS, "-I", B.CSRC, "-shared", os.path.join(HERE, "mlp_probe.cu"), "-o", so],
                   check=True)
    probe = ctypes.CDLL(so)
    rng = np.random.default_rng(2)
    X = torch.from_numpy(rng.standard_normal((512, Ln.K_PAD)).astype(np.float32)).cuda().bfloat16()
    T = torch.from_numpy(rng.standard_normal((512, 3)).astype(np.float32)).cuda()
    rows = torch.arange(128, dtype=torch.int32, device="cuda")
    net = Ln.ShellNet(Ln.init_params(3), batch_cap=128)
    loss = torch.zeros(1, device="cuda")
    before = net.params()
    assert probe.set_train_err(net.h, 1 << 7) == 0  # bit CUBE_ERR_TIMEOUT
    net.train_step(X, T, rows, 128, 1e-3, loss)
    torch.cuda.synchronize()
    with pytest.raises(CubeError):
        net.params()
    assert probe.set_train_err(net.h, 0) == 0
    np.testing.assert_array_equal(net.params(), before)
    net.train_step(X, T, rows, 128, 1e-3, loss)
    assert np.any(net.params() != before)
    net.close()
