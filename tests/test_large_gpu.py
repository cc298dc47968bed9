"""Transforms larger than one CTA (n = 32768 ... 2^20): the four-step kernels, against
the FP64 oracle and one another, and the scratch they share."""
import numpy as np
import pytest

from oracle import oracle, parity

pytestmark = pytest.mark.gpu


def _mf():
    import apogee_b200 as mf
    return mf


def noise(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("n", [32768, 65536, 131072, 262144])
def test_large_parity(n):
    mf = _mf()
    rng = np.random.default_rng(n + 1)
    nd, nt = 2, 3
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    z = oracle.correlate(D, H)
    for binsize, thr, win in [(n // 16, 0.0, None), (n // 64, 0.0, None), (4096, 0.0, None),
                              (n // 100 + 7, 0.0, (13, n - 5)),
                              (n // 8, 4.0 * np.sqrt(n), (n // 3, n)), (n, 0.0, None)]:
        out, cnt = f.run(binsize=binsize, threshold=thr, window=win, counts=True)
        bad = parity.compare(out["index"], out["value"], z, binsize, thr, win)
        assert not bad, (binsize, thr, win, bad[:3])
        np.testing.assert_array_equal(cnt, (out["index"] >= 0).sum(-1))


def test_largest_length():
    mf = _mf()
    n = 1 << 20
    rng = np.random.default_rng(3)
    D, H = noise(rng, (1, n)), noise(rng, (2, n))
    f = mf.MatchedFilter(n, 1, 2)
    f.set_data(D)
    f.set_templates(H)
    out = f.run(binsize=n // 256)
    assert not parity.compare(out["index"], out["value"], oracle.correlate(D, H), n // 256)


def test_large_known_lag_and_subrange():
    mf = _mf()
    n = 262144
    rng = np.random.default_rng(4)
    x = noise(rng, n)
    lags = (0, 1, 12345, n - 1)
    H = np.stack([x * np.exp(2j * np.pi * np.arange(n) * lag / n) for lag in lags]).astype(np.complex64)
    f = mf.MatchedFilter(n, 1, len(lags))
    f.set_data(x[None])
    f.set_templates(H)
    out = f.run(binsize=n)
    np.testing.assert_array_equal(out["index"][0, :, 0], lags)
    sub = f.run(binsize=n, templates=(1, 2))
    np.testing.assert_array_equal(sub["index"][0, :, 0], lags[1:3])


def test_large_too_many_bins_refused():
    mf = _mf()
    n = 65536
    f = mf.MatchedFilter(n, 1, 1)
    f.set_data(np.ones((1, n), np.complex64))
    f.set_templates(np.ones((1, n), np.complex64))
    with pytest.raises(ValueError):
        f.run(binsize=8)


def test_large_hierarchical_refine_is_flat():
    """Gate 0 refines every pair: the hierarchical result equals the flat one."""
    mf = _mf()
    n, nd, nt = 65536, 2, 3
    rng = np.random.default_rng(5)
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    flat = mf.MatchedFilter(n, nd, nt)
    hf = mf.HierarchicalFilter(n, nd, nt, band=n // 16, coarse="fp32")
    hf.set_coarse_threshold(0.0)
    for o in (flat, hf):
        o.set_data(D)
        o.set_templates(H)
    a = flat.run(binsize=n // 16).copy()
    b = hf.run(binsize=n // 16)
    np.testing.assert_array_equal(a, b)
    assert hf.stats == (nd * nt, nd * nt)


@pytest.mark.parametrize("n", [32768, 131072])
def test_large_run_series(n):
    """run_series for n > 16384: two-pass forward transforms of the blocks,
    then the two-pass filter, grouped by window (src/matchfilt.c:437-490)."""
    mf = _mf()
    rng = np.random.default_rng(n + 7)
    nt = 3
    H = noise(rng, (nt, n))
    series = rng.standard_normal(3 * n + n // 3).astype(np.float32)
    starts = np.array([0, n // 2, n, 2 * n, 3 * n])          # the last one runs past the end
    ws = np.array([n // 8, n // 8, 0, n // 8, n // 8])
    we = np.array([n, n, n - n // 8, n, n])
    f = mf.MatchedFilter(n, 2, nt)
    f.set_templates(H)
    bs = n // 32
    idx, val = f.run_series(series.astype(np.complex64), starts, ws, we, binsize=bs, raw=True)
    z = oracle.correlate(oracle.series_spectra(series, starts, n), H)
    for b in range(starts.size):
        bad = parity.compare(idx[b:b + 1], val[b:b + 1], z[b:b + 1], bs, 0.0,
                             (int(ws[b]), int(we[b])))
        assert not bad, (b, bad[:3])


@pytest.mark.parametrize("coarse", ["fp16x3", "bf16x3"])
@pytest.mark.parametrize("nd,nt,window", [(3, 5, None), (4, 160, (1000, 30000))])
def test_band_16384_tensor_core_coarse(coarse, nd, nt, window):
    """The split-precision tensor-core coarse pass at band 16384 (a four-step
    around the 512-point tensor-core pass, batches of 512 pairs): coarse
    maxima against FP64 over the widened coarse window, and a gated run whose
    fired rows are the flat filter's rows and whose dismissed rows are empty."""
    import apogee_b200 as mf
    n, band = 32768, 16384
    rng = np.random.default_rng(nd * 1000 + nt)
    D = (rng.standard_normal((nd, n)) + 1j * rng.standard_normal((nd, n))).astype(np.complex64)
    H = (rng.standard_normal((nt, n)) + 1j * rng.standard_normal((nt, n))).astype(np.complex64)
    hf = mf.HierarchicalFilter(n, nd, nt, band=band, coarse=coarse)
    hf.set_coarse_threshold(0.0)
    hf.set_data(D)
    hf.set_templates(H)
    cv = hf.coarse_values(window=window)
    cm = oracle.coarse_max(D, H, band, None, window)
    rel = np.abs(cv - cm) / cm
    assert rel.max() < 2e-5, rel.max()
    gate = float(np.quantile(cm, 0.7))
    hf.set_coarse_threshold(gate)
    bs = n // 16
    out = hf.run(binsize=bs, threshold=0.0, window=window).copy()
    flat = mf.MatchedFilter(n, nd, nt)
    flat.set_data(D)
    flat.set_templates(H)
    ref = flat.run(binsize=bs, threshold=0.0, window=window)
    fired = (out["index"] >= 0).any(-1)
    assert hf.last_refinements == int(fired.sum())
    np.testing.assert_array_equal(fired, cv >= gate)
    np.testing.assert_array_equal(out[fired], ref[fired])
    assert (out["index"][~fired] == -1).all() and (out["value"][~fired] == 0).all()


@pytest.mark.parametrize("n, nd, nt", [
    (32768, 1, 1),       # one pair: half an item
    (65536, 3, 141),     # odd pair count, data rows change inside items, more items than ring slots
    (131072, 2, 3),
    (262144, 2, 75),     # the ring of item slots is reused
    (524288, 1, 4),
])
@pytest.mark.parametrize("bins", ["even", "ragged", "one"])
def test_persistent_kernel_equals_two_pass(n, nd, nt, bins):
    """The persistent four-step kernel (two pairs per thread, items through a ring of
    scratch slots) against the two-pass kernels of the entry point without
    allocation: same arithmetic, same bits; run twice, the second run on the
    counters and records the first left behind."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(n + nt)
    D = torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    f = mf.MatchedFilter(n, nd, nt)
    _lib.check(L.mfb_set_cluster(f._plan, 0))
    f.set_data(D)
    f.set_templates(H)
    binsize, win = {"even": (n // 16, (0, n)), "ragged": (n // 50 + 3, (17, n - 9)),
                    "one": (n, (0, n))}[bins]
    for thr in (0.0, 3.3 * np.sqrt(n)):
        nb = L.mfb_nbins(n, binsize, *win)
        idx = torch.full((nd, nt, nb), -7, dtype=torch.int64, device="cuda")
        val = torch.zeros(nd, nt, nb, dtype=torch.complex64, device="cuda")
        cnt = torch.zeros(nd, nt, dtype=torch.int32, device="cuda")
        _lib.check(L.mfb_run_large_static(0, n, D.data_ptr(), nd, H.data_ptr(), nt, binsize, thr,
                                          *win, idx.data_ptr(), val.data_ptr(), cnt.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream))
        for _ in range(2):
            i2, v2 = f.run_device(binsize=binsize, threshold=thr, window=win)
            assert torch.equal(i2, idx) and torch.equal(v2, val)
        out, c2 = f.run(binsize=binsize, threshold=thr, window=win, counts=True)
        np.testing.assert_array_equal(c2, cnt.cpu().numpy())


def test_persistent_kernel_lists_and_streams():
    """Listed rows (odd count, arbitrary order, none) give the dense run's rows;
    runs of one plan enqueued on two streams do not disturb one another."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    n, nd, nt = 65536, 4, 60
    g = torch.Generator(device="cuda").manual_seed(9)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g))
    f.set_templates(torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g))
    ref_i, ref_v = f.run_device(binsize=n // 16)
    ref_w, _ = f.run_device(binsize=n // 64, threshold=800.0)
    torch.cuda.synchronize()
    rows = torch.from_numpy(np.random.default_rng(3).permutation(nd * nt)[:77].astype(np.int32)).cuda()
    for k in (0, 1, 77):
        idx = torch.full((nd * nt, 16), -7, dtype=torch.int64, device="cuda")
        val = torch.zeros(nd * nt, 16, dtype=torch.complex64, device="cuda")
        cnt = torch.tensor([k], dtype=torch.int32, device="cuda")
        f._bind_stream()
        _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), cnt.data_ptr(), 77, n // 16,
                                  0.0, 0, n, idx.data_ptr(), val.data_ptr(), None))
        r = rows[:k].long()
        assert torch.equal(idx[r], ref_i.view(-1, 16)[r]) and torch.equal(val[r], ref_v.view(-1, 16)[r])
        assert int((idx == -7).all(1).sum()) == nd * nt - k
    cnt = torch.tensor([78], dtype=torch.int32, device="cuda")
    assert L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), cnt.data_ptr(), 77, n // 16, 0.0, 0,
                          n, idx.data_ptr(), val.data_ptr(), None) < 0
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for i in range(6):
        with torch.cuda.stream(streams[i & 1]):
            got.append(f.run_device(binsize=n // 16) if i % 3 else f.run_device(binsize=n // 64, threshold=800.0))
    torch.cuda.synchronize()
    for i, (a, b) in enumerate(got):
        if i % 3:
            assert torch.equal(a, ref_i) and torch.equal(b, ref_v)
        else:
            assert torch.equal(a, ref_w)


def test_series_ring_grows_beyond_the_plan():
    """run_series over more blocks than the plan has data rows: the scratch grows,
    and the spectra and peaks stay those of the blocks."""
    mf = _mf()
    n, nt, blocks = 65536, 2, 40
    rng = np.random.default_rng(5)
    x = noise(rng, n // 2 * (blocks + 1))
    H = noise(rng, (nt, n))
    f = mf.MatchedFilter(n, 1, nt)
    f.set_templates(H)
    f.set_data(noise(rng, (1, n)))
    f.run(binsize=n)                          # sizes the ring for one pair of rows
    starts = np.arange(blocks) * (n // 2)
    out = f.run_series(x, starts, np.full(blocks, n // 4), np.full(blocks, 3 * n // 4), binsize=n // 8)
    for b in (0, 7, 39):
        D = np.fft.fft(x[starts[b]:starts[b] + n].astype(np.complex128) / n)
        z = oracle.correlate(D[None], H)
        assert not parity.compare(out["index"][b][None], out["value"][b][None], z, n // 8, 0.0,
                                  (n // 4, 3 * n // 4))


def test_run_that_gave_up_spoils_no_later_one():
    """A dependency wait that runs out (a count that is never reached; no GPU fault) leaves
    counters and records half-way.  The next runs start from zero all the same: a replay
    of a graph captured before, which no host call precedes, and a direct run."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    n, nd, nt = 65536, 3, 25
    g = torch.Generator(device="cuda").manual_seed(4)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g))
    f.set_templates(torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g))
    nb = 16
    idx = torch.empty(nd, nt, nb, dtype=torch.int64, device="cuda")
    val = torch.empty(nd, nt, nb, dtype=torch.complex64, device="cuda")
    other_i, other_v = torch.empty_like(idx), torch.empty_like(val)

    def run(i, v):
        f._bind_stream()
        return L.mfb_run(f._plan, 0, nd, 0, nt, n // nb, 0.0, 0, n, i.data_ptr(), v.data_ptr(), None)
    _lib.check(run(idx, val))
    torch.cuda.synchronize()
    ref_i, ref_v = idx.clone(), val.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _lib.check(run(idx, val))
    _lib.check(L.mfb_test_wait_limit(f._plan, 1))
    _lib.check(run(other_i, other_v))
    torch.cuda.synchronize()
    _lib.check(L.mfb_test_wait_limit(f._plan, -1))
    for _ in range(2):
        idx.fill_(-7)
        graph.replay()
        assert torch.equal(idx, ref_i) and torch.equal(val, ref_v)
    assert run(idx, val) < 0                     # reports the run that gave up
    idx.fill_(-7)
    _lib.check(run(idx, val))
    assert torch.equal(idx, ref_i) and torch.equal(val, ref_v)


def test_run_that_gave_up_is_reported():
    """run(), run_series(), a hierarchical run (direct, then its replayed graph) and a
    batch's wait() raise for the very run whose dependency wait ran out, and the next
    run is right."""
    mf = _mf()
    from apogee_b200 import _lib
    from apogee_b200.batch import BatchedFilter, Job
    L = _lib.lib()
    n, nd, nt = 65536, 2, 9
    rng = np.random.default_rng(8)
    D, H = noise(rng, (nd, n)), noise(rng, (nt, n))
    x = noise(rng, 2 * n)

    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    st, lo, hi = np.array([0, n // 2]), np.zeros(2, int), np.full(2, n)
    def series():
        return f.run_series(x, st, lo, hi, binsize=n // 4)
    def flat():
        f.set_data(D)
        return f.run(binsize=n // 16).copy()
    h = mf.HierarchicalFilter(n, nd, nt, band=8192, coarse="fp32")
    h.set_coarse_threshold(0.0)
    h.set_data(D)
    h.set_templates(H)
    def hier():
        return h.run(binsize=n // 16).copy()
    for call, plan, hook in ((flat, f._plan, L.mfb_test_wait_limit), (series, f._plan, L.mfb_test_wait_limit),
                             (hier, None, L.mfb_hier_test_wait_limit)):
        ref = call()
        p = plan if plan is not None else h._hplan
        _lib.check(hook(p, 1))
        for _ in range(3):                       # hier: direct, captured, replayed
            with pytest.raises(RuntimeError, match="timed out on a dependency"):
                call()
        _lib.check(hook(p, -1))
        for _ in range(3):
            np.testing.assert_array_equal(call(), ref)

    bf = BatchedFilter([Job(H, data=D, binsize=n // 16)], tune={n: {"dedicated": True}})
    bf.run()
    bf.wait()
    ref = bf.result(0).copy()
    _lib.check(L.mfb_test_wait_limit(bf._own[0]["plan"], 1))
    bf.run()
    with pytest.raises(RuntimeError, match="timed out on a dependency"):
        bf.wait()
    _lib.check(L.mfb_test_wait_limit(bf._own[0]["plan"], -1))
    bf.run()
    bf.wait()
    np.testing.assert_array_equal(bf.result(0), ref)
    bf.close()


def _held(make):
    """Device bytes that `make` leaves allocated, and what it returns."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    out = make()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return free - torch.cuda.mem_get_info()[0], out


def _plan(n, nd, nt, owner=None):
    import ctypes
    from apogee_b200 import _lib
    h = ctypes.c_void_p()
    if owner is None:
        _lib.check(_lib.lib().mfb_create(ctypes.byref(h), n, nd, nt, 0))
    else:
        _lib.check(_lib.lib().mfb_create_sharing(ctypes.byref(h), n, nd, nt, owner))
    return h


def _run_plan(p, n, nd, nt, nb):
    """One dense run on zeroed rows; its (idx, val)."""
    import torch
    from apogee_b200 import _lib
    L = _lib.lib()
    idx = torch.empty(nd * nt * nb, dtype=torch.int64, device="cuda")
    val = torch.empty(nd * nt * nb, dtype=torch.complex64, device="cuda")
    _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
    _lib.check(L.mfb_run(p, 0, nd, 0, nt, n // nb, 0.0, 0, n, idx.data_ptr(), val.data_ptr(), None))
    return idx, val


def test_scratch_is_what_the_runs_need():
    """Nothing is held for lists and small blocks at n = 32768; records follow the bins; a
    scratch that is outgrown is given back; a plan made to share holds none."""
    import torch
    from apogee_b200 import _lib
    import apogee_b200 as mf
    L = _lib.lib()
    MB = 1 << 20
    n = 32768
    rows = lambda nd, nt: (nd + nt) * n * 8
    _run_plan(_plan(n, 1, 1), n, 1, 1, 16)                       # constants of this length
    held, p = _held(lambda: _plan(n, 2, 32))
    assert held <= rows(2, 32) + 4 * MB
    L.mfb_destroy(p)
    held, h = _held(lambda: mf.HierarchicalFilter(n, 2, 300, band=16384, coarse="fp32"))
    held_p, p = _held(lambda: _plan(n, 2, 300))
    assert held_p <= rows(2, 300) + 213 * MB                     # rows, and records for 512 bins
    allocated, _ = _held(lambda: [_run_plan(p, n, 2, 300, nb)[0].sum().item() for nb in (1, 64, 512)])
    assert allocated <= 0                                        # no run at this length allocates
    L.mfb_destroy(p)
    del h

    n = 65536
    nd, nt = 2, 300
    def first():
        p = _plan(n, nd, nt)
        _run_plan(p, n, nd, nt, 16)
        return p
    first()                                                      # constants of this length
    base = (nd + nt) * n * 8
    held, p = _held(first)
    assert held <= base + 213 * MB
    grown, _ = _held(lambda: _run_plan(p, n, nd, nt, 4096)[0].sum().item())
    assert grown <= 60 * MB + 2 * nd * nt * 4096 * 16            # 2 x 27 MB of records, and the outputs
    held, q = _held(lambda: _plan(n, nd, nt, owner=p))
    assert held <= base + 4 * MB
    L.mfb_destroy(p)                                             # q keeps the scratch
    _run_plan(q, n, nd, nt, 16)
    L.mfb_destroy(q)


def test_plans_that_share_scratch():
    """Plans of different lengths on one scratch, interleaved on two streams and replayed
    from one graph, give what plans of their own give."""
    import torch
    from apogee_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(2)
    shapes = [(131072, 2, 3, 16), (32768, 5, 41, 64), (65536, 3, 50, 256), (262144, 1, 5, 16)]
    plans, alone, want = [], [], []
    for n, nd, nt, nb in shapes:
        D = torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g)
        H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
        pair = []
        for owner in (None, plans[0] if plans else None):
            p = _plan(n, nd, nt, owner)
            _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
            if n == 32768:
                _lib.check(L.mfb_set_cluster(p, 0))
            _lib.check(L.mfb_set_data(p, 0, nd, D.data_ptr()))
            _lib.check(L.mfb_set_templates(p, 0, nt, H.data_ptr()))
            pair.append(p)
        torch.cuda.synchronize()
        alone.append(pair[0])
        plans.append(pair[1])
        want.append(_run_plan(pair[0], n, nd, nt, nb))
    def all_runs():
        return [_run_plan(p, *s) for p, s in zip(plans, shapes)]
    def check(got):
        torch.cuda.synchronize()
        for (i, v), (wi, wv) in zip(got, want):
            assert torch.equal(i, wi) and torch.equal(v, wv)
    check(all_runs())
    check(all_runs()[::-1][::-1])
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for r in range(8):
        s = streams[r & 1]
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            got.append(_run_plan(plans[r % 4], *shapes[r % 4]))
    torch.cuda.synchronize()
    check(got[:4])
    check(got[4:])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = all_runs()
    for _ in range(2):
        for i, _v in got:
            i.fill_(-7)
        graph.replay()
        check(got)
    check(all_runs())
    for p in alone + plans:
        L.mfb_destroy(p)


def test_outgrown_scratch_of_a_captured_run_stays():
    """A graph captured before the scratch grew replays on what it was captured with."""
    import torch
    from apogee_b200 import _lib
    L = _lib.lib()
    n, nd, nt, nb = 65536, 1, 8, 16
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(60 * n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    p = _plan(n, nd, nt)
    _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
    _lib.check(L.mfb_set_data(p, 0, nd, x.data_ptr()))
    _lib.check(L.mfb_set_templates(p, 0, nt, H.data_ptr()))
    want = _run_plan(p, n, nd, nt, nb)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _run_plan(p, n, nd, nt, nb)
    st = np.arange(60, dtype=np.uint64) * n                      # 480 pairs of 1024 bins: everything grows
    lo, hi = np.zeros(60, np.uint64), np.full(60, n, np.uint64)
    idx = torch.empty(60 * nt * 1024, dtype=torch.int64, device="cuda")
    val = torch.empty(60 * nt * 1024, dtype=torch.complex64, device="cuda")
    _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
    _lib.check(L.mfb_run_series(p, x.data_ptr(), x.numel(), st.ctypes.data, lo.ctypes.data, hi.ctypes.data,
                                60, 0, nt, n // 1024, 0.0, idx.data_ptr(), val.data_ptr(), None))
    for _ in range(2):
        got[0].fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    L.mfb_destroy(p)


@pytest.mark.parametrize("n", [32768, 65536, 131072, 262144, 524288])
@pytest.mark.parametrize("binsize, win", [
    ("n/4096", (0, 1)),          # whole groups of a unit's neighbouring lags: one key per k1
    ("n/1024 + 1", (0, 1)),      # groups that straddle two bins
    ("n/3000", (0.013, 0.97)),   # and a window on no boundary
    ("3", (0.4, 0.4)),           # bins narrower than a group, in a short window
])
def test_many_bins(n, binsize, win):
    """Up to 4096 bins per pair, an odd pair count, at threshold 0 (every lag a candidate) and
    above: the persistent kernel's keys by k1 against the two-pass kernels' keys by bin."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    binsize = eval(binsize.replace("/", "//"), {"n": n})
    lo, hi = int(win[0] * n), int(win[1] * n)
    if lo == hi:
        lo, hi = lo + 5, lo + 5 + 3 * 4000 - 1
    nd, nt = 1, 3
    g = torch.Generator(device="cuda").manual_seed(n)
    D = torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    f = mf.MatchedFilter(n, nd, nt)
    _lib.check(L.mfb_set_cluster(f._plan, 0))
    f.set_data(D)
    f.set_templates(H)
    nb = L.mfb_nbins(n, binsize, lo, hi)
    assert 900 < nb <= 4096
    for thr in (0.0, 3.3 * np.sqrt(n)):
        idx = torch.full((nd, nt, nb), -7, dtype=torch.int64, device="cuda")
        val = torch.zeros(nd, nt, nb, dtype=torch.complex64, device="cuda")
        rc = L.mfb_run_large_static(0, n, D.data_ptr(), nd, H.data_ptr(), nt, binsize, thr, lo, hi,
                                    idx.data_ptr(), val.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
        _lib.check(rc)
        rows = torch.arange(nd * nt, dtype=torch.int32, device="cuda")   # lists take no other kernel
        count = torch.tensor([nd * nt], dtype=torch.int32, device="cuda")
        for _ in range(2):
            i2, v2 = torch.full_like(idx, -7), torch.zeros_like(val)
            f._bind_stream()
            _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), count.data_ptr(), nd * nt, binsize,
                                      thr, lo, hi, i2.data_ptr(), v2.data_ptr(), None))
            assert torch.equal(i2, idx) and torch.equal(v2, val)
            i2, v2 = f.run_device(binsize=binsize, threshold=thr, window=(lo, hi))
            assert torch.equal(i2, idx) and torch.equal(v2, val)


@pytest.mark.parametrize("n, nd, nt, nb, thr", [
    (65536, 1, 1, 50, 0.0),
    (32768, 1, 128, 50, 0.0),        # the last on clusters
    (32768, 1, 129, 50, 0.0),        # on the launches per batch
    (32768, 1, 65, 50, 600.0),       # in the persistent kernel
    (32768, 1, 96, 4090, 0.0),
    (65536, 1, 16, 4090, 0.0),       # 2^20 lags of many bins, and one pair more
    (65536, 1, 17, 4090, 0.0),
    (65536, 2, 64, 50, 0.0),         # 2^23 lags: the last on the launches per batch
    (65536, 3, 43, 50, 0.0),         # the first in the persistent kernel
    (65536, 1, 1, 4090, 900.0),
    (131072, 5, 7, 1024, 0.0),       # the edge on bins, either side and threshold
    (131072, 5, 7, 1025, 0.0),
    (131072, 5, 7, 1024, 1200.0),
    (131072, 5, 7, 1025, 1200.0),
    (262144, 1, 3, 300, 0.0),
    (524288, 2, 2, 16, 0.0),
    (1 << 20, 1, 1, 16, 0.0),        # any bins
    (1 << 20, 1, 2, 16, 3000.0),
    (1 << 20, 1, 3, 16, 0.0),
    (1 << 20, 1, 2, 1000, 0.0),
])
def test_short_runs(n, nd, nt, nb, thr):
    """Dense runs around the rule on short runs give the bits of the same rows listed (which
    always take the persistent kernel), direct, with counts and captured."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(n + nb)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g))
    f.set_templates(torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g))
    lo, hi = (0, n) if nb == 16 else (7, n - 30)
    binsize = n // 16 if nb == 16 else -(-(hi - lo) // nb)
    nb = L.mfb_nbins(n, binsize, lo, hi)
    shape = (nd, nt, nb)
    rows = torch.arange(nd * nt, dtype=torch.int32, device="cuda")
    count = torch.tensor([nd * nt], dtype=torch.int32, device="cuda")
    idx = torch.full(shape, -7, dtype=torch.int64, device="cuda")
    val = torch.zeros(shape, dtype=torch.complex64, device="cuda")
    f._bind_stream()
    _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), count.data_ptr(), nd * nt, binsize, thr,
                              lo, hi, idx.data_ptr(), val.data_ptr(), None))
    kw = dict(binsize=binsize, threshold=thr, window=(lo, hi))
    for _ in range(2):
        i, v = f.run_device(**kw)
        assert torch.equal(i, idx) and torch.equal(v, val)
    out, cnt = f.run(counts=True, **kw)
    np.testing.assert_array_equal(out["index"], idx.cpu().numpy())
    np.testing.assert_array_equal(cnt, (idx >= 0).sum(-1).cpu().numpy())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        i, v = f.run_device(**kw)
    for _ in range(2):
        i.fill_(-7)
        graph.replay()
        assert torch.equal(i, idx) and torch.equal(v, val)
    count.zero_()                                # an empty list writes nothing
    idx.fill_(-7)
    f._bind_stream()
    _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), count.data_ptr(), nd * nt, binsize, thr,
                              lo, hi, idx.data_ptr(), val.data_ptr(), None))
    assert (idx == -7).all()
    i, v = f.run_device(**kw)
    assert not (i == -7).any()


def test_outgrown_scratch_of_a_captured_forward_stays():
    """The same for a captured forward transform, which is all that a plan at n = 32768 with few
    pairs uses the scratch for."""
    import torch
    from apogee_b200 import _lib
    L = _lib.lib()
    n, nt = 32768, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(50 * n, dtype=torch.complex64, device="cuda", generator=g)
    st = np.arange(50, dtype=np.uint64) * n
    st_d = torch.from_numpy(st.astype(np.int64)).cuda()
    p = _plan(n, 1, nt)
    spec = torch.zeros(2, n, dtype=torch.complex64, device="cuda")

    def forward():
        _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
        _lib.check(L.mfb_forward(p, x.data_ptr(), x.numel(), st_d.data_ptr(), 2, spec.data_ptr()))
    forward()
    torch.cuda.synchronize()
    want = spec.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        forward()
    _lib.check(L.mfb_set_stream(p, torch.cuda.current_stream().cuda_stream))
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    _lib.check(L.mfb_set_templates(p, 0, nt, H.data_ptr()))
    lo, hi = np.zeros(50, np.uint64), np.full(50, n, np.uint64)
    rec = torch.empty(50 * nt * 16 * 2, dtype=torch.int64, device="cuda")
    _lib.check(L.mfb_run_series_records(p, x.data_ptr(), x.numel(), st.ctypes.data, lo.ctypes.data, hi.ctypes.data,
                                        50, 0, nt, n // 16, 0.0, rec.data_ptr(), None))   # the scratch grows
    for _ in range(2):
        spec.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(spec, want)
    L.mfb_destroy(p)


@pytest.mark.parametrize("binsize, win, thr", [
    ("n/16", None, 0.0),             # every warp's rows lie in one bin
    ("n/16", None, 3.6),
    ("n", None, 0.0),
    ("n/50 + 3", (17, -9), 0.0),     # bins shared by lanes at random
    ("n/50 + 3", (17, -9), 3.6),
    ("n/3000", (5, -1), 3.6),        # more bins than a unit sees lags of
])
def test_longest_transform(binsize, win, thr):
    """n = 2^20, where a row spans two warps and both passes exchange across the CTA: 37 pairs
    (more items than ring slots, the last one half empty), dense against the same rows
    listed and, for two pairs, against FP64; each twice, on the counters and records that the
    first run left."""
    import torch
    mf = _mf()
    from apogee_b200 import _lib
    L = _lib.lib()
    n, nd, nt = 1 << 20, 1, 37
    binsize = eval(binsize.replace("/", "//"), {"n": n})
    lo, hi = (0, n) if win is None else (win[0], n + win[1])
    g = torch.Generator(device="cuda").manual_seed(20)
    D = torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g)
    H = torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g)
    thr *= np.sqrt(n)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(D)
    f.set_templates(H)
    nb = L.mfb_nbins(n, binsize, lo, hi)
    rows = torch.randperm(nt, device="cuda", generator=g).to(torch.int32)
    count = torch.tensor([nt], dtype=torch.int32, device="cuda")
    for _ in range(2):
        i, v = f.run_device(binsize=binsize, threshold=thr, window=(lo, hi))
        li, lv = torch.full_like(i, -7), torch.zeros_like(v)
        f._bind_stream()
        _lib.check(L.mfb_run_rows(f._plan, 0, nd, 0, nt, rows.data_ptr(), count.data_ptr(), nt, binsize, thr,
                                  lo, hi, li.data_ptr(), lv.data_ptr(), None))
        assert torch.equal(i, li) and torch.equal(v, lv)
        sel = [0, nt - 1]
        z = oracle.correlate(D.cpu().numpy(), H[sel].cpu().numpy())
        got = i[:, sel].cpu().numpy()
        assert (got >= 0).any()
        assert not parity.compare(got, v[:, sel].cpu().numpy(), z, binsize, thr, (lo, hi))


def test_two_streams_at_32768():
    """Blocks of more pairs than the cluster kernel takes, enqueued on two streams, share the
    plan's scratch one after another."""
    import torch
    mf = _mf()
    n, nd, nt = 32768, 2, 300
    g = torch.Generator(device="cuda").manual_seed(7)
    f = mf.MatchedFilter(n, nd, nt)
    f.set_data(torch.randn(nd, n, dtype=torch.complex64, device="cuda", generator=g))
    f.set_templates(torch.randn(nt, n, dtype=torch.complex64, device="cuda", generator=g))
    want = [f.run_device(binsize=n // 16), f.run_device(binsize=n // 60 + 1, threshold=500.0)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for k in range(8):
        with torch.cuda.stream(streams[k & 1]):
            got.append(f.run_device(binsize=n // 16) if k % 3 else f.run_device(binsize=n // 60 + 1, threshold=500.0))
    torch.cuda.synchronize()
    for k, (i, v) in enumerate(got):
        wi, wv = want[0 if k % 3 else 1]
        assert torch.equal(i, wi) and torch.equal(v, wv)
