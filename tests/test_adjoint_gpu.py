"""The adjoint kernel behind peak_values: gradients of peak values and
|value|^2 with respect to data and template spectra, and through the torch
template generator to (alpha, t_c), against a torch.fft dense-correlation
gradient in FP64 and FP64 central finite differences (step 1e-6)."""
import numpy as np
import pytest

from apogee_b200 import synthetic

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def dense_loss(D, H, idx, weights=None):
    """FP64 reference: sum over reported bins of |z|^2, or Re(conj(w) z), with
    z the dense torch.fft correlation gathered at the given lags."""
    torch = _torch()
    n = D.shape[-1]
    z = torch.fft.ifft(D[:, None, :] * torch.conj(H[None, :, :]), dim=-1) * n
    zb = torch.gather(z, 2, idx.clamp(min=0))
    mask = idx >= 0
    if weights is None:
        return ((zb.real ** 2 + zb.imag ** 2) * mask).sum()
    return ((torch.conj(weights) * zb).real * mask).sum()


def workload(n, nd, nt, seed):
    rng = np.random.default_rng(seed)
    H = synthetic.template_bank(n, nt, rng)
    D = synthetic.noise_spectra(n, nd, rng)
    for d in range(0, nd, 3):
        synthetic.inject(D, H, d, int(rng.integers(nt)), int(rng.integers(n)), 8.0)
    return D.astype(np.complex64), H


def reference_grads(D32, H32, idx, weights=None):
    torch = _torch()
    D = D32.detach().to(torch.complex128).requires_grad_(True)
    H = H32.detach().to(torch.complex128).requires_grad_(True)
    dense_loss(D, H, idx, weights).backward()
    return D.grad.resolve_conj(), H.grad.resolve_conj()


def assert_close(ours, ref, rel_l2=2e-5, rel_max=2e-4):
    """FP32 adjoint against the FP64 gradient: relative L2 error and largest
    elementwise error relative to the largest gradient component."""
    torch = _torch()
    ours = ours.to(torch.complex128)
    diff = ours - ref
    scale = ref.abs().max().item()
    assert scale > 0
    assert (diff.norm() / ref.norm()).item() <= rel_l2, (diff.norm() / ref.norm()).item()
    assert diff.abs().max().item() <= rel_max * scale, diff.abs().max().item() / scale


@pytest.mark.parametrize("n,nd,nt,binsize,thr", [
    (16384, 8, 256, 1024, 0.0),      # the differentiable-peaks workload
    (1024, 3, 40, 16, 0.0),          # many bins per pair
    (4096, 1, 7, 4096, 4.5),         # one bin, thresholded, split over templates
    (65536, 2, 3, 4096, 0.0),        # two-pass forward
])
def test_power_gradient_matches_dense_fp64(n, nd, nt, binsize, thr):
    torch = _torch()
    from apogee_b200.adjoint import peak_values
    Dn, Hn = workload(n, nd, nt, seed=n + nd)
    D = torch.from_numpy(Dn).cuda().requires_grad_(True)
    H = torch.from_numpy(Hn).cuda().requires_grad_(True)
    idx, val, power = peak_values(D, H, binsize, threshold=thr)
    power.sum().backward()
    if thr > 0:
        assert (idx < 0).any() and (idx >= 0).any()
    gD, gH = reference_grads(D, H, idx)
    assert_close(D.grad, gD)
    assert_close(H.grad, gH)


def test_value_gradient_and_forward_values():
    torch = _torch()
    import apogee_b200 as mf
    from apogee_b200.adjoint import peak_values
    n, nd, nt, binsize = 16384, 4, 32, 1024
    Dn, Hn = workload(n, nd, nt, seed=5)
    D = torch.from_numpy(Dn).cuda().requires_grad_(True)
    H = torch.from_numpy(Hn).cuda().requires_grad_(True)
    idx, val, power = peak_values(D, H, binsize)
    from oracle import oracle, parity
    bad = parity.compare(idx.cpu().numpy(), val.detach().cpu().numpy(),
                         oracle.correlate(Dn, Hn), binsize)
    assert not bad, bad[:3]
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(Dn)
    f.set_templates(Hn)
    ref = f.run(binsize=binsize)
    np.testing.assert_array_equal(idx.cpu().numpy(), ref["index"])
    np.testing.assert_array_equal(val.detach().cpu().numpy(), ref["value"])
    g = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn(val.shape, dtype=torch.complex64, device="cuda", generator=g)
    (torch.conj(w) * val).real.sum().backward()
    gD, gH = reference_grads(D, H, idx, w.to(torch.complex128))
    assert_close(D.grad, gD)
    assert_close(H.grad, gH)


def test_directional_finite_difference_fp64():
    torch = _torch()
    from apogee_b200.adjoint import peak_values
    n, nd, nt, binsize = 16384, 8, 256, 1024
    Dn, Hn = workload(n, nd, nt, seed=9)
    D = torch.from_numpy(Dn).cuda().requires_grad_(True)
    H = torch.from_numpy(Hn).cuda().requires_grad_(True)
    idx, val, power = peak_values(D, H, binsize)
    power.sum().backward()
    g = torch.Generator(device="cuda").manual_seed(2)
    VD = torch.randn(D.shape, dtype=torch.complex128, device="cuda", generator=g)
    VH = torch.randn(H.shape, dtype=torch.complex128, device="cuda", generator=g)
    D64, H64 = D.detach().to(torch.complex128), H.detach().to(torch.complex128)
    h = 1e-6
    with torch.no_grad():
        fd = (dense_loss(D64 + h * VD, H64 + h * VH, idx)
              - dense_loss(D64 - h * VD, H64 - h * VH, idx)).item() / (2 * h)
    an = ((torch.conj(D.grad.to(torch.complex128)) * VD).real.sum()
          + (torch.conj(H.grad.to(torch.complex128)) * VH).real.sum()).item()
    assert abs(fd - an) <= 1e-4 * abs(an), (fd, an)


def test_template_parameter_gradient():
    """d sum|peak|^2 / d(alpha, t_c) through the torch template generator and the
    adjoint, against FP64 central finite differences of the dense loss."""
    torch = _torch()
    from apogee_b200.adjoint import peak_values
    n, nd, nt, binsize = 16384, 8, 16, 1024
    rng = np.random.default_rng(11)
    alpha0 = rng.uniform(1e2, 1e4, size=nt)
    tc0 = rng.uniform(0, n, size=nt)
    Dn = synthetic.noise_spectra(n, nd, rng)
    H0 = synthetic.template_bank_torch(n, torch.tensor(alpha0), torch.tensor(tc0)).numpy()
    for d in range(nd):
        synthetic.inject(Dn, H0, d, d % nt, int(rng.integers(n)), 10.0)
    D = torch.from_numpy(Dn.astype(np.complex64)).cuda()
    alpha = torch.tensor(alpha0, device="cuda", requires_grad=True)
    tc = torch.tensor(tc0, device="cuda", requires_grad=True)
    H = synthetic.template_bank_torch(n, alpha, tc).to(torch.complex64)
    idx, val, power = peak_values(D, H, binsize)
    power.sum().backward()
    D64 = D.to(torch.complex128)

    def loss(a, t):
        with torch.no_grad():
            return dense_loss(D64, synthetic.template_bank_torch(n, a, t), idx).item()
    h = 1e-6
    a0, t0 = alpha.detach(), tc.detach()
    fd_a = np.empty(nt)
    fd_t = np.empty(nt)
    for i in range(nt):
        e = torch.zeros(nt, dtype=torch.float64, device="cuda")
        e[i] = h
        fd_a[i] = (loss(a0 + e, t0) - loss(a0 - e, t0)) / (2 * h)
        fd_t[i] = (loss(a0, t0 + e) - loss(a0, t0 - e)) / (2 * h)
    ga, gt = alpha.grad.cpu().numpy(), tc.grad.cpu().numpy()
    np.testing.assert_allclose(ga, fd_a, rtol=0, atol=1e-3 * np.abs(fd_a).max())
    np.testing.assert_allclose(gt, fd_t, rtol=0, atol=1e-3 * np.abs(fd_t).max())


def _adjoint_direct(n, nd, nt, nb, seed, peaks):
    """mfb_adjoint on random lags; both gradients and the FP64 sums they
    stand for, with the sum of absolute terms behind every output."""
    import torch
    from apogee_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(seed)
    def cplx(*shape):
        return torch.randn(*shape, dtype=torch.complex64, device="cuda", generator=g)
    D, H, gz = cplx(nd, n), cplx(nt, n), cplx(nd, nt, nb)
    idx = torch.randint(0, n, (nd, nt, nb), device="cuda", generator=g)
    idx[torch.rand(nd, nt, nb, device="cuda", generator=g) >= peaks] = -1
    gd, gh = torch.full_like(D, float("nan")), torch.full_like(H, float("nan"))
    _lib.check(_lib.lib().mfb_adjoint(0, n, D.data_ptr(), nd, H.data_ptr(), nt, nb, idx.data_ptr(),
                                      gz.data_ptr(), gd.data_ptr(), gh.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream))
    live = idx >= 0
    g64 = torch.where(live, gz.to(torch.complex128), torch.zeros((), dtype=torch.complex128, device="cuda"))
    wd, wh = torch.zeros(nd, n, dtype=torch.complex128, device="cuda"), []
    ad = torch.zeros(nd, n, dtype=torch.float64, device="cuda")
    ah = []
    D64, H64 = D.to(torch.complex128), H.to(torch.complex128)
    for t in range(nt):
        s = torch.zeros(nd, n, dtype=torch.complex128, device="cuda")
        s.scatter_add_(1, idx[:, t].clamp(min=0), g64[:, t])
        u = torch.fft.fft(s, dim=1)
        a = g64[:, t].abs().sum(1, keepdim=True)
        wd += u * H64[t]
        ad += a * H64[t].abs()
        wh.append((u.conj() * D64).sum(0))
        ah.append((a * D64.abs()).sum(0))
    return (gd, wd, ad), (gh, torch.stack(wh), torch.stack(ah))


@pytest.mark.parametrize("n, nd, nt, nb, peaks", [
    (64, 3, 70, 1, 1.0),        # 4 frequencies per row: 64 own rows per CTA, a ragged last one
    (64, 65, 2, 64, 0.5),       # every lag a bin: many lists per row
    (256, 7, 3, 33, 1.0),       # one entry more than a list
    (512, 2, 5, 32, 0.9),       # lists exactly full
    (1024, 9, 2, 100, 0.7),     # four own rows per CTA, several lists per row
    (4096, 1, 1, 1, 1.0),       # one row, one entry
    (4096, 5, 200, 16, 0.05),   # rows without a peak among the summed ones
    (8192, 2, 3, 300, 1.0),     # a row's lists in several rounds
    (1024, 2, 8, 4, 1.0),       # 8 splits: atomics alone
    (1024, 2, 9, 4, 1.0),       # 9: clusters of eight, seven blocks of them without rows
    (2048, 3, 872, 4, 1.0),     # as many clusters as fit a wave
    (4096, 17, 5, 4, 1.0),      # one tile too many for clusters
    (16384, 3, 40, 16, 0.0),    # no peak at all
    (1 << 20, 1, 2, 3, 1.0),    # the longest transform
])
def test_adjoint_kernel_edges(n, nd, nt, nb, peaks):
    """Both gradients against FP64 at the edges of the kernel's lists, rounds
    and row blocks.  Every output is a sum of g * row * W terms: two twiddles
    within 2 ulp and three products (12 roundings of at most 2^-24 each),
    a 16-point transform (8), and as many additions as a row has entries and
    there are rows -- the bound below, relative to the sum of |g| |row|."""
    for got, want, scale in _adjoint_direct(n, nd, nt, nb, n + nb, peaks):
        bound = (24 + nb + max(nd, nt)) * 2.0 ** -24 * scale
        err = (got.to(want.dtype) - want).abs()
        assert bool((err <= bound + 1e-30).all()), (n, nd, nt, nb, float((err / scale.clamp(min=1e-30)).max()))


@pytest.mark.parametrize("direct, n, nd, nt, nb, peaks", [
    (1, 64, 1, 600, 1, 1.0),        # half a warp of frequencies, splits summed by clusters
    (1, 64, 3, 9, 64, 0.7),         # nine splits: two clusters, most without rows
    (1, 512, 5, 8, 33, 1.0),        # eight splits: atomics alone
    (1, 1024, 2, 100, 4, 0.01),     # rows without a peak
    (1, 4096, 7, 1, 20, 1.0),       # one summed row
    (1, 16384, 19, 3, 1, 1.0),      # two own rows per thread, the last CTA's second one missing
    (1, 16384, 38, 3, 1, 0.5),      # four
    (1, 16384, 77, 16, 1, 1.0),     # eight, as many summed rows as the rule allows
    (1, 1 << 18, 4, 2, 2, 1.0),
    (0, 64, 65, 140, 64, 0.5),      # 64 own rows per CTA, a second block of one row
    (0, 256, 70, 60, 33, 1.0),      # one entry more than a list
    (0, 512, 40, 20, 32, 0.9),      # lists exactly full
    (0, 1024, 9, 12, 100, 0.7),     # four own rows per CTA, several lists per row
    (0, 16384, 2, 8, 20, 1.0),      # 8 splits: atomics alone
    (0, 16384, 2, 9, 20, 1.0),      # 9: clusters of eight
    (0, 4096, 17, 5, 16, 1.0),      # one tile too many for clusters
])
def test_both_adjoint_kernels_at_their_edges(direct, n, nd, nt, nb, peaks):
    """As test_adjoint_kernel_edges (its bound holds for both: the direct form has two
    twiddles and their product, three products and as many additions), each shape on the
    kernel that the rule gives its data gradient."""
    import ctypes
    import torch
    from apogee_b200 import _lib
    out = (ctypes.c_int64 * 5)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _lib.check(_lib.lib().mfb_adjoint_plan(n, nd, nt, nb, sms, out))
    if sms == 148:
        assert out[4] == direct
    for got, want, scale in _adjoint_direct(n, nd, nt, nb, n + nb, peaks):
        bound = (24 + nb + max(nd, nt)) * 2.0 ** -24 * scale
        err = (got.to(want.dtype) - want).abs()
        assert bool((err <= bound + 1e-30).all()), (n, nd, nt, nb, float((err / scale.clamp(min=1e-30)).max()))


@pytest.mark.parametrize("n, nb", [(1024, 4), (16384, 64)])
def test_row_without_a_peak_adds_nothing(n, nb):
    """A NaN row that no pair reports a peak for leaves the gradients finite, on both
    kernels."""
    import torch
    from apogee_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(n)
    nd, nt = 4, 12
    D = torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    H[5] = float("nan")
    idx = torch.randint(0, n, (nd, nt, nb), device="cuda", generator=g)
    idx[:, 5] = -1
    gz = torch.randn(nd, nt, nb, dtype=torch.complex64, device="cuda", generator=g)
    gd, gh = torch.full_like(D, float("nan")), torch.full_like(H, float("nan"))
    _lib.check(_lib.lib().mfb_adjoint(0, n, D.data_ptr(), nd, H.data_ptr(), nt, nb, idx.data_ptr(),
                                      gz.data_ptr(), gd.data_ptr(), gh.data_ptr(),
                                      torch.cuda.current_stream().cuda_stream))
    assert torch.isfinite(torch.view_as_real(gd)).all()
    assert (gh[5] == 0).all() and torch.isfinite(torch.view_as_real(gh)).all()
