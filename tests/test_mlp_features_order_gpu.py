"""learned.features without a stream: the rows are there when it returns, whatever torch's stream does next with them."""
import pytest

pytestmark = pytest.mark.gpu


def test_rows_are_there_on_return(gpu):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.layout import Layout, build_image
    L = Layout(ng=128, nnt=2, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.uniform_random(128 ** 3, 128.0, 7), L)
    rho, idx, xp, _ = Ln.device_image(img, gpu)
    own = torch.as_tensor(img.active, device=gpu)
    X = Ln.features(L, rho, idx, xp, img.n_used)  # allocates what the next call finds
    torch.cuda.synchronize()
    first = torch.empty_like(X)
    del X
    torch.cuda.synchronize()
    X = Ln.features(L, rho, idx, xp, img.n_used)
    first.copy_(X)  # on torch's stream, without waiting
    torch.cuda.synchronize()
    assert torch.equal(first, X)
    assert bool((X[own].float().abs().amax(1) > 0).all())
