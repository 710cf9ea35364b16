"""learned.features without a stream: the rows are there when it returns, whatever torch's stream does next with them.
With one the call waits for nothing."""
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


def test_a_given_stream_is_not_waited_for(gpu, monkeypatch):
    import torch
    from cube2_b200 import ic
    from cube2_b200 import learned as Ln
    from cube2_b200.layout import Layout, build_image
    L = Layout(ng=32, nnt=1, nns=1, ratio_cs=4, ngb=4, app=0.1)
    img = build_image(*ic.uniform_random(32 ** 3, 32.0, 7), L)
    rho, idx, xp, _ = Ln.device_image(img, gpu)
    want = Ln.features(L, rho, idx, xp, img.n_used)
    s = torch.cuda.Stream()

    def waits(*a, **k):
        raise AssertionError("the call waited")
    with monkeypatch.context() as m, torch.cuda.stream(s):
        m.setattr(torch.cuda, "synchronize", waits)
        m.setattr(torch.cuda.Stream, "synchronize", waits)
        X = Ln.features(L, rho, idx, xp, img.n_used, stream=s)
    s.synchronize()
    # the density by particle: float atomics, which may turn single BF16 inputs
    assert float((X.float() - want.float()).abs().max()) <= 2.0 ** -6
