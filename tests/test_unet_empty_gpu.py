"""kw_unet_flip_weights of no weights does nothing, as an empty loop does."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cout,cin", [(0, 8), (8, 0), (0, 0)])
def test_flip_no_weights(cout, cin):
    import torch
    from kwave_gb300 import _lib

    w = torch.ones(72, dtype=torch.bfloat16, device="cuda")
    wt = torch.full((72,), 2.0, dtype=torch.bfloat16, device="cuda")
    _lib.check(_lib.lib().kw_unet_flip_weights(w.data_ptr(), wt.data_ptr(), cout, cin, None))
    torch.cuda.synchronize()
    assert bool((wt == 2).all())
