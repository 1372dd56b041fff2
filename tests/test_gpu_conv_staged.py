"""The staged forms of the corrector's convolution kernels at the sizes where
they change: boxes too wide for two stages, ragged last tiles, many tiles a
block, output addresses that are not 32-byte aligned; the fused input gradient
against the separate kernels and the Adam list against single calls, both bit
for bit.  Forward and weight gradients against the float64 oracle with the
bounds of test_gpu_conv.py."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from multicellular_phase_field_active_gel_organoids_b200 import capi  # noqa: E402
from oracle import conv_oracle as co  # noqa: E402
from tests.test_gpu_conv import P, dev, run_fwd  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,cin,cout", [(1, 3, 700, 32, 32), (2, 2, 660, 32, 16), (1, 1, 1, 16, 32),
                                            (5, 31, 61, 32, 32), (40, 30, 30, 16, 32)])
def test_forward_and_weight_gradient(B, H, W, cin, cout):
    rng = np.random.default_rng(B + H + W)
    x = co.pad(co.bf16(rng.normal(size=(B, H, W, cin))))
    w = co.bf16(rng.normal(size=(cout, 9, cin)) / np.sqrt(9 * cin))
    b = rng.normal(size=cout).astype(np.float32).astype(np.float64)
    y, pre = run_fwd(x, w, b, True, B, H, W, cin, cout)
    z = co.conv_fwd(x, w, b)
    ref = co.gelu(z)
    assert np.max(np.abs(y[:, 1:-1, 1:-1, :] - ref)) <= 1e-2 * np.abs(ref).max()
    assert np.max(np.abs(pre[:, 1:-1, 1:-1, :] - z)) <= 1e-2 * np.abs(z).max()
    for halo in (y[:, 0], y[:, -1], y[:, :, 0], y[:, :, -1]):
        assert not np.any(halo)
    dz = co.bf16(rng.normal(size=(B, H, W, cout)))
    xd, dzd = dev(x, torch.float32).to(torch.bfloat16), dev(co.pad(dz), torch.float32).to(torch.bfloat16)
    dw = torch.zeros((cout, 9, cin), dtype=torch.float32, device="cuda")
    db = torch.zeros(cout, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    capi.check(capi.lib().pfag_conv3x3_wgrad(P(xd), P(dzd), P(dw), P(db), B, H, W, cin, cout, P(err), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    rdw, rdb = co.conv_wgrad(x, dz)
    assert np.max(np.abs(dw.cpu().numpy() - rdw)) <= 1e-3 * np.abs(rdw).max()
    assert np.max(np.abs(db.cpu().numpy() - rdb)) <= 1e-3 * np.abs(rdb).max()


def test_forward_into_half_aligned_output():
    """An output 16 but not 32 bytes past an aligned address takes the narrow stores."""
    B, H, W, c = 2, 9, 33, 32
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.zeros((B, H + 2, W + 2, c), dtype=torch.bfloat16, device="cuda")
    x[:, 1:-1, 1:-1] = torch.randn((B, H, W, c), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((c, 9, c), generator=g, device="cuda") / 17).to(torch.bfloat16)
    b = torch.randn(c, generator=g, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for off in (0, 8):
        flat = torch.zeros(x.numel() + 16, dtype=torch.bfloat16, device="cuda")
        y = flat[off:off + x.numel()]
        capi.check(capi.lib().pfag_conv3x3(P(x), P(w), P(b), P(y), None, B, H, W, c, c, 1, P(err), None))
        torch.cuda.synchronize()
        outs.append(y.clone())
        assert not flat[off + x.numel():].any() and not flat[:off].any()
    assert int(err.item()) == 0 and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16), (16, 16)])
@pytest.mark.parametrize("B,H,W", [(2, 5, 7), (3, 31, 30), (1, 2, 700)])
@pytest.mark.parametrize("gelu_on", [0, 1])
def test_fused_input_gradient_equals_the_separate_kernels(B, H, W, cin, cout, gelu_on):
    g = torch.Generator(device="cuda").manual_seed(B * 100 + H + gelu_on)

    def padded(c):
        t = torch.zeros((B, H + 2, W + 2, c), dtype=torch.bfloat16, device="cuda")
        t[:, 1:-1, 1:-1] = torch.randn((B, H, W, c), generator=g, device="cuda").to(torch.bfloat16)
        return t

    L = capi.lib()
    dz, pre = padded(cout), padded(cin)
    w = (torch.randn((cout, 9, cin), generator=g, device="cuda") / 17).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    wt = torch.zeros((cin, 9, cout), dtype=torch.bfloat16, device="cuda")
    zb = torch.zeros(cin, device="cuda")
    da, ref, got = torch.zeros_like(pre), torch.zeros_like(pre), torch.zeros_like(pre)
    capi.check(L.pfag_conv_flip(P(w), P(wt), cin, cout, None))
    capi.check(L.pfag_conv3x3(P(dz), P(wt), P(zb), P(da), None, B, H, W, cout, cin, 0, P(err), None))
    capi.check(L.pfag_conv_act_bwd(P(da), P(pre), P(ref), B, H, W, cin, gelu_on, None))
    capi.check(L.pfag_conv3x3_dgrad(P(dz), P(w), P(pre) if gelu_on else None, P(got), B, H, W, cin, cout, gelu_on,
                                    P(err), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert ref.abs().max() > 0 and torch.equal(got, ref)


def test_adam_list_equals_single_calls():
    g = torch.Generator(device="cuda").manual_seed(1)
    L = capi.lib()
    sizes = [1, 255, 256, 9217, 32]
    sets = []
    for _ in range(2):
        g.manual_seed(1)
        sets.append([[torch.randn(n, generator=g, device="cuda") for n in sizes] for _ in range(3)]
                    + [[torch.rand(n, generator=g, device="cuda") for n in sizes]])
    pb = [[torch.zeros(n, dtype=torch.bfloat16, device="cuda") for n in sizes] for _ in range(2)]
    p, gr, m, v = sets[0]
    for k, n in enumerate(sizes):
        capi.check(L.pfag_adam(P(p[k]), P(gr[k]), P(m[k]), P(v[k]), P(pb[0][k]) if k else None, None, n, 1e-3, 0.9,
                               0.999, 1e-8, 3, None))
    p2, gr2, m2, v2 = sets[1]
    arr = lambda ts: (ctypes.c_void_p * len(sizes))(*[t.data_ptr() if t is not None else None for t in ts])  # noqa: E731
    capi.check(L.pfag_adam_list(len(sizes), arr(p2), arr(gr2), arr(m2), arr(v2), arr([None] + pb[1][1:]),
                                (ctypes.c_int * len(sizes))(*sizes), 1e-3, 0.9, 0.999, 1e-8, 3, None))
    torch.cuda.synchronize()
    for a, b in zip(sets[0] + [pb[0]], sets[1] + [pb[1]]):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
    with pytest.raises(capi.PfagError):
        capi.check(L.pfag_adam_list(17, None, None, None, None, None, None, 1e-3, 0.9, 0.999, 1e-8, 1, None))


@pytest.mark.parametrize("B,offset", [(2, 0), (2, 2), (2, 8), (400, 0)])
def test_loss_gradient_addresses(B, offset):
    """The output gradient at addresses that are not 16-byte aligned, and more
    boxes than blocks; bounds of test_gpu_conv.py."""
    H, W, C = 5, 6, 16
    rng = np.random.default_rng(B + offset)
    out = co.pad(co.bf16(rng.normal(size=(B, H, W, C))))
    tgt = rng.normal(size=(B, H, W, 2)).astype(np.float32)
    od, td = dev(out, torch.float32).to(torch.bfloat16), dev(tgt, torch.float32)
    buf = torch.ones(od.numel() + 16, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    dst = ctypes.c_void_p(buf.data_ptr() + offset)
    capi.check(capi.lib().pfag_conv_mse(P(od), P(td), dst, P(loss), B, H, W, C, 2, 0.5, None))
    torch.cuda.synchronize()
    d = out[:, 1:-1, 1:-1, :2] - tgt
    assert abs(float(loss.item()) - float((d * d).sum())) <= 1e-4 * float((d * d).sum())
    h = buf.float().cpu().numpy()
    k = offset // 2
    g = h[k:k + od.numel()].reshape(out.shape)
    assert np.max(np.abs(g[:, 1:-1, 1:-1, :2] - d)) <= 1e-2 * np.abs(d).max()
    assert not np.any(g[:, 1:-1, 1:-1, 2:]) and not np.any(g[:, 0])
    assert (h[:k] == 1).all() and (h[k + od.numel():] == 1).all()
