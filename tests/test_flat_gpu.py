"""Flat matched filter on the device vs the FP64 oracle and the reference's
own outputs (tests/golden).  Bar: oracle/parity.py."""
import os

import numpy as np
import pytest

from oracle import oracle, parity

pytestmark = pytest.mark.gpu


def _mf():
    import apogee_b200 as mf
    return mf


def noise(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def check(filt, D, H, binsize, threshold=0.0, window=None, **kw):
    out = filt.run(binsize=binsize, threshold=threshold, window=window, **kw)
    z = oracle.correlate(D, H)
    bad = parity.compare(out["index"], out["value"], z, binsize, threshold, window)
    assert not bad, bad[:5]
    return out


SIZES = [64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384]


@pytest.mark.parametrize("n", SIZES)
def test_parity_all_lengths(n):
    mf = _mf()
    rng = np.random.default_rng(n)
    D, H = noise(rng, (3, n)), noise(rng, (5, n))
    f = mf.MatchedFilter(n, 3, 5)
    f.set_data(D)
    f.set_templates(H)
    for binsize, thr, win in [(n, 0.0, None), (n // 16, 0.0, None), (n // 64 or 1, 0.0, None),
                              (17, 0.0, (3, n - 5)), (1, 0.0, None),
                              (n // 4, 3.0 * np.sqrt(n), (1, n)), (n + 3, 0.0, (n // 3, n))]:
        check(f, D, H, binsize, thr, win)


def test_matches_reference_golden(golden_dir):
    """Same inputs as the reference engine saw; same peaks (near ties aside)."""
    mf = _mf()
    g = np.load(os.path.join(golden_dir, "flat.npz"))
    for c in range(int(g["ncases"])):
        n, nd, nt, seed, bs, thr, w0, w1 = g["c%d_par" % c]
        n, nd, nt, bs = int(n), int(nd), int(nt), int(bs)
        win = None if w0 < 0 else (int(w0), int(w1))
        D, H = g["c%d_D" % c], g["c%d_H" % c]
        f = mf.MatchedFilter(n, nd, nt)
        f.set_data(D)
        f.set_templates(H)
        out, cnt = f.run(binsize=bs, threshold=float(thr), window=win, counts=True)
        z = oracle.correlate(D, H)
        assert not parity.compare(out["index"], out["value"], z, bs, float(thr), win)
        ri = g["c%d_idx" % c]
        diff = out["index"] != ri
        m = np.abs(z)
        for pos in zip(*np.nonzero(diff)):
            a, b = out["index"][pos], ri[pos]
            assert a >= 0 and b >= 0, (c, pos, a, b)
            assert abs(m[pos[:-1] + (a,)] - m[pos[:-1] + (b,)]) <= 1e-5 * m[pos[:-1] + (b,)]
        np.testing.assert_array_equal(cnt, g["c%d_cnt" % c])


def test_exact_ties_report_lowest_lag(golden_dir):
    """DC-only products tie at every lag (tests/test_cpu_single_peak.py)."""
    mf = _mf()
    g = np.load(os.path.join(golden_dir, "ties.npz"))
    filters = {}
    for c in range(int(g["ncases"])):
        n, lo, hi, bs, thr = g["c%d_par" % c]
        n, lo, hi, bs = int(n), int(lo), int(hi), int(bs)
        if n not in filters:
            data = np.zeros((3, n), np.complex64)
            data[:, 0] = [3 + 4j, -5j, 0]
            tm = np.zeros((5, n), np.complex64)
            tm[:, 0] = 1
            f = mf.MatchedFilter(n, 3, 5)
            f.set_data(data)
            f.set_templates(tm)
            filters[n] = f
        out = filters[n].run(binsize=bs, threshold=float(thr), window=(lo, hi))
        np.testing.assert_array_equal(out["index"], g["c%d_idx" % c])
        np.testing.assert_array_equal(out["value"], g["c%d_val" % c])


def test_period_four_tie_keeps_earliest():
    """Exact period-four correlation [0, 4, 4, 0] (test_cpu_single_peak.py:38-50)."""
    mf = _mf()
    n = 64
    data = np.zeros(n, np.complex64)
    data[[0, n // 4, 3 * n // 4]] = [2, -1 - 1j, -1 + 1j]
    f = mf.MatchedFilter(n, 1, 17)
    f.set_data(data[None, :])
    f.set_templates(np.ones((17, n), np.complex64))
    for window in [(0, 4), (1, 4), (4, 9), (5, 8), (63, 64)]:
        out = f.run(window=window, binsize=n)
        eligible = [k for k in range(*window) if k % 4 in (1, 2)]
        np.testing.assert_array_equal(out["index"], eligible[0] if eligible else -1)
        np.testing.assert_array_equal(out["value"], 4 if eligible else 0)


def test_known_lag():
    mf = _mf()
    n = 4096
    rng = np.random.default_rng(1)
    x = noise(rng, n)
    f = mf.MatchedFilter(n, 1, 5)
    f.set_data(x[None, :])
    lags = (0, 1, 37, n // 2, n - 1)
    f.set_templates(np.stack([x * np.exp(2j * np.pi * np.arange(n) * lag / n) for lag in lags])
                    .astype(np.complex64))
    out = f.run(binsize=n)
    np.testing.assert_array_equal(out["index"][0, :, 0], lags)


def test_self_correlation_and_flat_spectrum():
    mf = _mf()
    n = 1024
    rng = np.random.default_rng(2)
    h = noise(rng, n)
    f = mf.MatchedFilter(n, 1, 1)
    f.set_data(h[None])
    f.set_templates(h[None])
    out = f.run(binsize=n)
    want = float(np.sum(np.abs(h.astype(np.complex128)) ** 2))
    assert out["index"][0, 0, 0] == 0
    assert abs(abs(out["value"][0, 0, 0]) - want) <= 1e-5 * want
    g = mf.MatchedFilter(512, 1, 1)
    g.set_data(np.ones((1, 512), np.complex64))
    g.set_templates(np.ones((1, 512), np.complex64))
    m = np.abs(g.run(binsize=1)["value"][0, 0])
    assert abs(m[0] - 512) <= 1e-5 * 512 and m[1:].max() < 1e-3 * 512


def test_zero_inputs_report_nothing():
    mf = _mf()
    n = 4096
    f = mf.MatchedFilter(n, 2, 2)
    f.set_data(np.zeros((2, n), np.complex64))
    f.set_templates(np.zeros((2, n), np.complex64))
    out, cnt = f.run(binsize=256, counts=True)
    assert (out["index"] == -1).all() and (out["value"] == 0).all() and (cnt == 0).all()


def test_amplitudes_and_subnormals():
    mf = _mf()
    n = 1024
    rng = np.random.default_rng(3)
    base = noise(rng, (1, n))
    f = mf.MatchedFilter(n, 1, 1)
    f.set_templates(base)
    for scale in (1e-12, 1e-6, 1.0, 1e6, 1e12):
        D = (base * np.float32(scale)).astype(np.complex64)
        f.set_data(D)
        check(f, D, base, 128)


def test_nan_isolated_to_its_pair():
    mf = _mf()
    n = 1024
    rng = np.random.default_rng(4)
    D, H = noise(rng, (2, n)), noise(rng, (2, n))
    D[1, 5] = np.nan
    f = mf.MatchedFilter(n, 2, 2)
    f.set_data(D)
    f.set_templates(H)
    out = f.run(binsize=256)
    z = oracle.correlate(D[:1], H)
    assert not parity.compare(out["index"][:1], out["value"][:1], z, 256)


def test_window_subrange_and_raw():
    mf = _mf()
    n, nd, nt = 4096, 4, 3
    rng = np.random.default_rng(5)
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    full = f.run(binsize=1024, window=(500, 3500)).copy()
    assert ((full["index"] >= 500) & (full["index"] < 3500)).all()
    sub = f.run(binsize=1024, window=(500, 3500), data=(1, 2), templates=(0, 2))
    np.testing.assert_array_equal(sub["index"], full["index"][1:3, 0:2])
    np.testing.assert_array_equal(sub["value"], full["value"][1:3, 0:2])
    idx, val = f.run(binsize=1024, window=(500, 3500), raw=True)
    np.testing.assert_array_equal(idx, full["index"])
    np.testing.assert_array_equal(val, full["value"])


def test_threshold_is_strict_and_counts():
    mf = _mf()
    n = 256
    d = np.zeros((1, n), np.complex64)
    d[0, 0] = 3 + 4j
    t = np.zeros((1, n), np.complex64)
    t[0, 0] = 1
    f = mf.MatchedFilter(n, 1, 1)
    f.set_data(d)
    f.set_templates(t)
    for thr, expect in ((4.99, 4), (5.0, 0), (0.0, 4), (-1.0, 4)):
        out, cnt = f.run(binsize=64, threshold=thr, counts=True)
        assert cnt[0, 0] == expect


def test_single_template_and_data_setters():
    mf = _mf()
    n = 1024
    rng = np.random.default_rng(6)
    D, H = noise(rng, (2, n)), noise(rng, (3, n))
    f = mf.MatchedFilter(n, 2, 3)
    with pytest.raises(ValueError):
        f.run(binsize=n)                      # no data yet
    for i in range(2):
        f.set_data(D[i], index=i)
    with pytest.raises(ValueError):
        f.run(binsize=n)                      # no templates yet
    for i in range(3):
        f.set_templates(H[i], index=i)
    check(f, D, H, 256)
    with pytest.raises(IndexError):
        f.set_data(D[0], index=2)
    with pytest.raises(ValueError):
        f.set_data(np.zeros((2, 100), np.complex64))


def test_argument_errors():
    mf = _mf()
    with pytest.raises(ValueError):
        mf.MatchedFilter(1000, 1, 1)
    with pytest.raises(ValueError):
        mf.MatchedFilter(4096, 0, 1)
    f = mf.MatchedFilter(4096, 1, 1)
    f.set_data(np.zeros((1, 4096), np.complex64))
    f.set_templates(np.zeros((1, 4096), np.complex64))
    with pytest.raises(ValueError):
        f.run(binsize=0)
    with pytest.raises(ValueError):
        f.run(window=(10, 10))
    with pytest.raises(ValueError):
        f.run(data=(0, 2))


def test_torch_device_inputs_match_host_inputs():
    import torch
    mf = _mf()
    n = 2048
    rng = np.random.default_rng(7)
    D, H = noise(rng, (2, n)), noise(rng, (4, n))
    f = mf.MatchedFilter(n, 2, 4)
    f.set_data(torch.from_numpy(D).cuda())
    f.set_templates(torch.from_numpy(H).cuda())
    a = f.run(binsize=128).copy()
    f.set_data(D)
    f.set_templates(H)
    b = f.run(binsize=128)
    np.testing.assert_array_equal(a, b)
    idx, val = f.run_device(binsize=128)
    np.testing.assert_array_equal(idx.cpu().numpy(), b["index"])
    np.testing.assert_array_equal(val.cpu().numpy(), b["value"])


def test_batch_independence():
    """A pair's result does not depend on the rest of the batch."""
    mf = _mf()
    n, nd, nt = 4096, 5, 7
    rng = np.random.default_rng(8)
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    full = f.run(binsize=512).copy()
    g = mf.MatchedFilter(n, 1, 1)
    g.set_data(D[3:4])
    g.set_templates(H[5:6])
    one = g.run(binsize=512)
    np.testing.assert_array_equal(one[0, 0], full[3, 5])


def _same_up_to_near_ties(i1, i2, z):
    """Indices equal except where the two lags' FP64 magnitudes are within
    1e-5 relative (either kernel may then report either lag)."""
    diff = np.nonzero(i1 != i2)
    for pos in zip(*diff):
        a, b = i1[pos], i2[pos]
        assert a >= 0 and b >= 0, pos
        za, zb = abs(z[pos[:-1]][a]), abs(z[pos[:-1]][b])
        assert abs(za - zb) <= 1e-5 * max(za, zb), (pos, a, b, za, zb)


@pytest.mark.parametrize("nd,nt,binsize,threshold", [
    (16, 1024, 256, 0.0),     # the benchmark block
    (5, 77, 512, 3.0),        # odd nt, thresholded
    (3, 1, 768, 0.0),         # one template: every pair on its own data row; a short last bin
    (1, 3, 4096, 2.0),        # fewer pairs than slots, one bin
    (3, 1, 64, 0.0),          # 64 bins of a quarter block: the general kernel either way
])
def test_packed_kernel_matches_one_pair_kernel_and_oracle(nd, nt, binsize, threshold):
    """n = 4096, bins of whole 256-lag blocks: the kernel that mfb_set_packed switches on
    (flatw_kernel) must meet the oracle's bar and equal the general kernel bit
    for bit (dense, listed and record output, counts: both form their twiddles
    with the same operations); listed rows equal the dense run's rows bit for bit.
    Bins off the grid run on the general kernel whatever the switch says."""
    import torch
    import apogee_b200 as mf
    from apogee_b200 import _lib
    n = 4096
    rng = np.random.default_rng(nd * 100 + nt)
    D = noise(rng, (nd, n))
    H = noise(rng, (nt, n))
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    L = _lib.lib()
    out = {}
    for packed in (0, 1):
        _lib.check(L.mfb_set_packed(f._plan, packed))
        r, c = f.run(binsize=binsize, threshold=threshold, counts=True)
        ri, rv = f.run(binsize=binsize, threshold=threshold, raw=True)
        out[packed] = (r.copy(), c.copy(), ri.copy(), rv.copy())
        np.testing.assert_array_equal(out[packed][0]["index"], out[packed][2])
        np.testing.assert_array_equal(out[packed][0]["value"], out[packed][3])
        np.testing.assert_array_equal(out[packed][1], (out[packed][2] >= 0).sum(-1))
    for t0 in range(0, nt, 128):
        z = oracle.correlate(D, H[t0:t0 + 128])
        for packed in (0, 1):
            r = out[packed][0][:, t0:t0 + 128]
            bad = parity.compare(r["index"], r["value"], z, binsize, threshold)
            assert not bad, (packed, bad[:3])
        _same_up_to_near_ties(out[0][2][:, t0:t0 + 128], out[1][2][:, t0:t0 + 128], z)
    np.testing.assert_array_equal(out[0][2], out[1][2])
    np.testing.assert_array_equal(out[0][3], out[1][3])
    # listed rows in arbitrary order, an odd count
    rows = np.random.default_rng(7).permutation(nd * nt)[: max(1, (nd * nt) // 2) | 1]
    rows_d = torch.as_tensor(rows.astype(np.int32), device="cuda")
    cnt_d = torch.tensor([rows.size], dtype=torch.int32, device="cuda")
    nb = -(-n // binsize)
    _lib.check(L.mfb_set_packed(f._plan, 1))
    f._bind_stream()
    idx = torch.full((nd * nt * nb,), -7, dtype=torch.int64, device="cuda")
    val = torch.zeros(nd * nt * nb, dtype=torch.complex64, device="cuda")
    _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows_d.data_ptr(), cnt_d.data_ptr(),
                              rows.size, binsize, threshold, 0, n, idx.data_ptr(),
                              val.data_ptr(), None))
    torch.cuda.synchronize()
    got_i = idx.cpu().numpy().reshape(nd * nt, nb)
    got_v = val.cpu().numpy().reshape(nd * nt, nb)
    np.testing.assert_array_equal(got_i[rows], out[1][2].reshape(nd * nt, nb)[rows])
    np.testing.assert_array_equal(got_v[rows], out[1][3].reshape(nd * nt, nb)[rows])
    untouched = np.setdiff1d(np.arange(nd * nt), rows)
    assert (got_i[untouched] == -7).all()


@pytest.mark.parametrize("n", [512, 1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("nd, nt, blocks, win", [
    (1, 1, 16, None),            # one pair: most pair slots have none
    (3, 5, 1, None),             # 15 pairs, data rows change between them
    (2, 301, 1, (4, 12)),        # a window of whole blocks (block-wise series filtering)
    (5, 7, 3, (1, 16)),          # bins of three blocks
    (1, 2, 8, (0, 1)),           # one block
])
def test_block_bins_kernel_is_bit_identical(n, nd, nt, blocks, win):
    """Bins and window in whole blocks of n/16 lags (the kernel whose exchanges
    stay within half-warps where they can) against flat_kernel: same bits,
    dense and listed; and against the FP64 oracle.  Thresholds: every bin
    reports, some do (z has deviation 2 sqrt(n) per component), none does."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(nd * 1000 + nt + n)
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    block = n // 16
    binsize = blocks * block
    win = None if win is None else (win[0] * block, win[1] * block)
    lo, hi = win or (0, n)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    z = oracle.correlate(D, H[:8])
    for thr in (0.0, 5.5 * np.sqrt(n), 1e3 * n):
        _lib.check(L.mfb_set_packed(f._plan, 1))
        out, cnt = f.run(binsize=binsize, threshold=thr, window=win, counts=True)
        out, cnt = out.copy(), cnt.copy()
        assert not parity.compare(out["index"][:, :8], out["value"][:, :8], z, binsize, thr, win)
        rows = torch.from_numpy(rng.permutation(nd * nt)[: nd * nt // 2 + 1].astype(np.int32)).cuda()
        count = torch.tensor([rows.numel()], dtype=torch.int32, device="cuda")
        nb = out.shape[2]
        idx = torch.full((nd * nt, nb), -7, dtype=torch.int64, device="cuda")
        val = torch.zeros(nd * nt, nb, dtype=torch.complex64, device="cuda")
        _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), count.data_ptr(), rows.numel(),
                                  binsize, thr, lo, hi, idx.data_ptr(), val.data_ptr(), None))
        r = rows.long().cpu().numpy()
        np.testing.assert_array_equal(idx.cpu().numpy()[r], out["index"].reshape(-1, nb)[r])
        np.testing.assert_array_equal(val.cpu().numpy()[r], out["value"].reshape(-1, nb)[r])
        _lib.check(L.mfb_set_packed(f._plan, 0))
        ref, rcnt = f.run(binsize=binsize, threshold=thr, window=win, counts=True)
        np.testing.assert_array_equal(out["index"], ref["index"])
        np.testing.assert_array_equal(out["value"], ref["value"])
        np.testing.assert_array_equal(cnt, rcnt)


@pytest.mark.parametrize("n, band", [(2048, 512), (4096, 1024), (8192, 2048), (8192, 4096), (16384, 8192),
                                     (32768, 16384), (1024, 256)])
def test_fp32_coarse_values_vs_fp64(n, band):
    """The FP32 gate pass at every band length, whole and partial windows, odd pair
    counts: coarse maxima against FP64.  Bound: the transform's FP32 error scales
    with its output's deviation (log2(band) stages of 2^-23 against a root mean
    square over the band), and keys drop five mantissa bits of |z|^2 (2^-19 of |z|)."""
    mf = _mf()
    rng = np.random.default_rng(band)
    nd, nt = 3, 7
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    P = (np.abs(H) ** 2).mean(0).astype(np.float32)
    hf = mf.HierarchicalFilter(n, nd, nt, band=band, coarse="fp32")
    hf.set_reference(P)
    hf.set_coarse_threshold(1.0)
    hf.set_data(D)
    hf.set_templates(H)
    f = float(np.float32(P[:band].astype(np.float64).sum() / P.astype(np.float64).sum()))
    R = n // band
    for window in (None, (n // 3, n // 2), (0, R)):
        lo, hi = (0, n) if window is None else window
        cs, ce = max(0, lo // R - 1), min(band, -(-hi // R))
        for d in range(nd):
            z = np.fft.ifft(D[d, :band].astype(np.complex128) * np.conj(H[:, :band]), axis=1) * band / np.sqrt(f)
            want = np.abs(z[:, cs:ce]).max(1)
            got = hf.coarse_values(window=window)[d]
            rms = np.sqrt((np.abs(z) ** 2).mean(1))
            assert (np.abs(got - want) <= 2.0 ** -19 * want + np.log2(band) * 2.0 ** -23 * 4 * rms).all()


@pytest.mark.parametrize("n", [64, 256, 1024, 2048, 8192, 16384])
@pytest.mark.parametrize("win", [None, (3, -5)])
def test_threshold_skips_only_pairs_without_candidates(n, win):
    """Above a threshold a warp whose points are all below it skips the per-bin
    reduction: one loud pair among quiet ones (in one warp with it where
    several pairs share a warp), bins on and off the 32-lag grid, many bins."""
    mf = _mf()
    rng = np.random.default_rng(n)
    D, H = noise(rng, (3, n)), noise(rng, (9, n))
    D[1] += (2.0 * H[4] * np.exp(-2j * np.pi * np.arange(n) * (n // 3) / n)).astype(np.complex64)
    w = None if win is None else (win[0], n + win[1])
    f = mf.MatchedFilter(n, 3, 9)
    f.set_data(D)
    f.set_templates(H)
    thr = float(n)
    for binsize in (n // 8, n // 16 + 1, max(1, n // 128)):
        out = check(f, D, H, binsize, thr, w)
        assert (out["index"][1, 4] >= 0).any()
        assert (out["index"] >= 0).any(-1).sum() < 27


@pytest.mark.parametrize("n", [64, 128, 256, 1024, 4096, 8192])
@pytest.mark.parametrize("thr", [0.0, 4.0])
def test_few_items_give_the_same_bits(n, thr):
    """Runs of up to two CTAs per SM (n = 8192: one) take flat_kernel's form with more
    registers: at the line, one pair past it and in pieces, general bins, against each other."""
    import torch
    mf = _mf()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = (2 if n <= 4096 else 1) * sms * max(1, 4096 // n)   # pairs that fill those CTAs
    g = torch.Generator(device="cuda").manual_seed(n)
    nt = line + 1
    D = torch.randn(1, n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    f = mf.MatchedFilter(n, 1, nt)
    f.set_data(D)
    f.set_templates(H)
    kw = dict(binsize=n // 5 + 1, threshold=thr * np.sqrt(n), window=(1, n - 2))
    whole = f.run_device(**kw)
    for parts in ((0, line), (line, 1), (5, 33)):
        i, v = f.run_device(templates=parts, **kw)
        t = slice(parts[0], parts[0] + parts[1])
        assert torch.equal(i, whole[0][:, t]) and torch.equal(v, whole[1][:, t])
    i, v = whole[0].cpu().numpy(), whole[1].cpu().numpy()
    z = oracle.correlate(D.cpu().numpy(), H[:8].cpu().numpy())
    assert not parity.compare(i[:, :8], v[:, :8], z, n // 5 + 1, thr * np.sqrt(n), (1, n - 2))
