"""pfag_conv3x3_wgrad does not read the halo rows of dz: with NaN there the
gradients match the float64 oracle as with zeros (bounds of test_gpu_conv.py),
on one tile, ragged last tiles, the one-stage form and on a dx that
pfag_conv3x3_dgrad wrote into a buffer nobody zeroed.  And the widths at which
the kernels go from two stages to one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from multicellular_phase_field_active_gel_organoids_b200 import capi  # noqa: E402
from oracle import conv_oracle as co  # noqa: E402
from tests import test_gpu_conv_staged as staged  # noqa: E402
from tests.test_gpu_conv import P, dev  # noqa: E402

pytestmark = pytest.mark.gpu


def wgrad(x, dz, B, H, W, cin, cout):
    dw = torch.zeros((cout, 9, cin), dtype=torch.float32, device="cuda")
    db = torch.zeros(cout, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    capi.check(capi.lib().pfag_conv3x3_wgrad(P(x), P(dz), P(dw), P(db), B, H, W, cin, cout, P(err), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return dw.cpu().numpy(), db.cpu().numpy()


@pytest.mark.parametrize("B,H,W,cin,cout", [(1, 1, 1, 16, 16), (2, 5, 7, 16, 32), (3, 31, 30, 32, 32),
                                            (2, 2, 500, 32, 16)])
def test_halo_rows_of_dz_are_not_read(B, H, W, cin, cout):
    rng = np.random.default_rng(B + H + W)
    x = co.pad(co.bf16(rng.normal(size=(B, H, W, cin))))
    dz = co.bf16(rng.normal(size=(B, H, W, cout)))
    dzp = co.pad(dz)
    dzp[:, 0] = dzp[:, -1] = np.nan
    dw, db = wgrad(dev(x, torch.float32).to(torch.bfloat16), dev(dzp, torch.float32).to(torch.bfloat16), B, H, W, cin,
                   cout)
    rdw, rdb = co.conv_wgrad(x, dz)
    assert np.max(np.abs(dw - rdw)) <= 1e-3 * np.abs(rdw).max()
    assert np.max(np.abs(db - rdb)) <= 1e-3 * np.abs(rdb).max()


def test_weight_gradient_of_an_input_gradient_in_a_fresh_buffer():
    B, H, W, c0, c1, c2 = 2, 9, 21, 16, 32, 16          # c0 -> c1 -> c2
    g = torch.Generator(device="cuda").manual_seed(4)

    def padded(c):
        t = torch.zeros((B, H + 2, W + 2, c), dtype=torch.bfloat16, device="cuda")
        t[:, 1:-1, 1:-1] = torch.randn((B, H, W, c), generator=g, device="cuda").to(torch.bfloat16)
        return t

    x, dz, pre = padded(c0), padded(c2), padded(c1)
    w = (torch.randn((c2, 9, c1), generator=g, device="cuda") / 17).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dx = torch.full_like(pre, float("nan"))
    capi.check(capi.lib().pfag_conv3x3_dgrad(P(dz), P(w), P(pre), P(dx), B, H, W, c1, c2, 1, P(err), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    inner = dx[:, 1:-1, 1:-1].float().cpu().numpy()
    assert np.isfinite(inner).all() and not dx[:, 1:-1, 0].any() and not dx[:, 1:-1, -1].any()
    dw, db = wgrad(x, dx, B, H, W, c0, c1)
    rdw, rdb = co.conv_wgrad(x.float().cpu().numpy(), inner)
    assert np.max(np.abs(dw - rdw)) <= 1e-3 * np.abs(rdw).max()
    assert np.max(np.abs(db - rdb)) <= 1e-3 * np.abs(rdb).max()


@pytest.mark.parametrize("W,cin,cout", [(477, 32, 16), (478, 32, 16), (597, 32, 32), (598, 32, 32), (633, 32, 16),
                                        (634, 32, 16), (1021, 16, 32), (1022, 16, 32), (1397, 16, 32), (1398, 16, 32),
                                        (1433, 16, 16), (1434, 16, 16)])
def test_widths_beside_the_change_of_stages(W, cin, cout):
    """The widest boxes of the two-stage forms and the narrowest of the one-stage
    ones (weight gradient 477 and 1021, forward the others)."""
    staged.test_forward_and_weight_gradient(1, 2, W, cin, cout)
