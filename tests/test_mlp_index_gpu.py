"""Storage indices of the copies that the learned shell's kick lists have 32 bits without a sign, so images of 2^31 copies
and more keep theirs; more than 2^32 are refused before anything is read or allocated."""
import os
import re

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_listed_index_is_unsigned():
    with open(os.path.join(HERE, "..", "cube2_b200", "csrc", "mlp.cu")) as f:
        text = f.read()
    assert "__uint_as_float((unsigned)(base + l))" in text
    readers = re.findall(r"p\.vp \+ 3 \* \(int64_t\)(\w+)\((?:q|p\.list\[i\])\.w\)", text)
    assert readers == ["__float_as_uint"] * 2
    # what is written and read back, at the ends of the range
    for i in (0, 1, 2 ** 31 - 1, 2 ** 31, 2 ** 32 - 1):
        w = np.array([i], np.int64).astype(np.uint32).view(np.float32)
        assert int(w.view(np.uint32)[0]) == i


@pytest.mark.gpu
def test_more_copies_are_refused(gpu):
    import torch
    from cube2_b200 import learned as Ln
    from cube2_b200.kick import CUBE_PM3_PERIODIC, CubeError, FineKick
    from cube2_b200.layout import Layout
    L = Layout(ng=32, nnt=1, nns=1, ratio_cs=4, ngb=4, app=0.1)
    FineKick(L, pm3_mode=CUBE_PM3_PERIODIC).configure()
    net = Ln.ShellNet(Ln.init_params(4), batch_cap=16)
    z = torch.zeros(4096, device=gpu)
    with pytest.raises(CubeError) as e:
        net.kick(z, z, z, 2 ** 32, z, 1.0, 1.0, 1.0)
    assert e.value.status == 1  # CUBE_ERR_INVALID
    net.close()
