"""The sweep at the edges of its tiling, against the oracle's emd_1d
(emd_ref.py:108-156): a warp tile is 32 runs of 8 float32 or 4 float64
samples, each warp of a task owns whole runs of its CTA's segment, and rows
that do not start on 32 bytes are read and written by element."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

from eemd4cuda_b200 import emd_par as M  # noqa: E402

# one sample to one side and the other of a run, a tile (128 and 256), a
# warp's share of 4 and 5 warps, and lengths that leave rows misaligned
LENGTHS = [127, 128, 129, 255, 256, 257, 511, 513, 1025, 1283, 2047, 2050, 4099]


def rows_of(lengths, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in lengths:
        t = np.arange(n, dtype=float)
        out.append(np.sin(2 * np.pi * t / 23.0) + 0.4 * np.sin(2 * np.pi * t / 6.1) + 0.3 * rng.standard_normal(n))
    return out


def end_rows():
    """Few knots: every interval of most tiles is clipped at the signal's ends;
    the last row has a single maximum (a constant upper envelope)."""
    n = 3001
    t = np.arange(n, dtype=float)
    one = np.minimum(np.sin(2 * np.pi * t / 700.0), 0.5)
    one += 0.7 * np.exp(-((t - 1575.0) / 30.0) ** 2)
    return [np.sin(2 * np.pi * t / 1300.0), np.sin(2 * np.pi * (t + 200) / 420.0) + 1e-4 * t, one]


def check(rows, tol, **kw):
    from oracle import emd_oracle as O
    from test_gpu_parity import engine_log, max_imf_err, oracle_log, raw_run

    dtype = kw.get("dtype", np.float64)
    rows = [r.astype(dtype).astype(np.float64) for r in rows]
    args = dict(tau=0.0, max_sifts=kw["max_sifts"], max_imf=kw["max_imf"], end=kw["end"])
    res = raw_run(None, x=np.concatenate(rows), lengths=[len(r) for r in rows], trial_count=1, exact=False,
                  dtype=dtype, config=kw["config"], **args)
    for k, row in enumerate(rows):
        imfs, resid, st = O.emd_1d(row, record_knots=True, **args)
        assert int(res["nmode"][k]) == st["n_modes"], len(row)
        assert engine_log(res, k) == oracle_log(st), len(row)
        scale = np.abs(row).max()
        assert max_imf_err(res["imfs"][k][:st["n_modes"]], imfs, scale) <= tol, len(row)
        assert np.max(np.abs(res["resid"][k] - resid)) <= tol * scale * max(1, st["n_modes"]), len(row)


@pytest.mark.parametrize("end", ["natural", "mirror"])
@pytest.mark.parametrize("cta_warps", [4, 5])
@pytest.mark.parametrize("csize", [1, 2])
def test_tile_edges_float64(end, cta_warps, csize):
    """Six sifts of up to six IMFs: knot counts of every sift equal, values
    within the seam-window solve's 1e-9 of max|x|."""
    lengths = LENGTHS if csize == 1 else [n for n in LENGTHS if n >= 256]
    cfg = M.EngineConfig(cluster_size=csize, cta_warps=cta_warps)
    check(rows_of(lengths, 11), 1e-9, max_sifts=6, max_imf=6, end=end, config=cfg)


@pytest.mark.parametrize("end", ["natural", "mirror"])
@pytest.mark.parametrize("cta_warps", [4, 5])
def test_tile_edges_float32(end, cta_warps):
    """One sift, so that no float32 rounding can move a knot: the envelopes'
    coefficients and Horner steps are rounded to 2^-24 of terms of the order
    of ten max|x| at most, which stays within 1e-5 of max|x|."""
    cfg = M.EngineConfig(cluster_size=1, cta_warps=cta_warps)
    check(rows_of(LENGTHS, 12), 1e-5, max_sifts=1, max_imf=1, end=end, dtype=np.float32, config=cfg)


@pytest.mark.parametrize("end", ["natural", "mirror"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("csize", [1, 8])
def test_clipped_intervals(end, dtype, csize):
    """Long stretches before the first and after the last knot, and an
    envelope of a single knot (bounds as above); with eight CTAs the few knots
    of a solve pass lie in more segments than are staged piece by piece."""
    cfg = M.EngineConfig(cluster_size=csize, cta_warps=4)
    check(end_rows(), 1e-9 if dtype == np.float64 else 1e-5, max_sifts=1, max_imf=1, end=end, dtype=dtype,
          config=cfg)


def density_rows():
    """Float32 runs of 8 samples with one, two, three and four knots, and slow
    rows in which single runs (at a tile's start, middle and end) have up to
    eight: tiles on both sides of the sparse store's bound, one next to the other."""
    n = 1541
    t = np.arange(n, dtype=float)
    out = [np.sin(2 * np.pi * (t + 0.3) / p) * (1 + 0.2 * np.cos(t / 97.0)) for p in (16.3, 8.1, 7.9, 5.2, 4.1)]
    for at in (512, 640, 764, 1019):
        fast = np.where((t >= at) & (t < at + 9), 1.0, 0.0) * np.cos(np.pi * t) * (1 + 0.01 * (t - at))
        out.append(np.sin(2 * np.pi * t / 61.7) + fast)
    return out


@pytest.mark.parametrize("end", ["natural", "mirror"])
def test_knot_densities_float32(end):
    """Bound as in test_tile_edges_float32; the fast runs' envelopes stay of
    the order of max|x| as their extrema alternate about the slow one."""
    cfg = M.EngineConfig(cluster_size=1, cta_warps=4)
    check(density_rows(), 1e-5, max_sifts=1, max_imf=1, end=end, dtype=np.float32, config=cfg)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1000, 1001, 1003, 4099])
def test_row_alignment_changes_nothing(dtype, n):
    """The caller's IMF rows on and off the 32-byte grid (sifted in a second
    scratch there), rows of the workspace padded to it, and the unpadded rows
    of a workspace of the bare size: the same IMFs and residuals bit for bit."""
    torch = pytest.importorskip("torch")
    from eemd4cuda_b200 import _lib as L

    E, M_ = 3, 4
    x = np.concatenate(rows_of([n], n) * E) + 0.1 * np.random.default_rng(n).standard_normal(E * n)
    xd = torch.from_numpy(x.astype(dtype)).cuda()
    p = M.make_params(dtype=dtype, noise_mode=L.EEMD_NOISE_PREPERTURBED, tau=0.25, max_sifts=9, max_imf=M_)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    got = []
    for shift in (0, 1):
        buf = torch.zeros((E * M_ * n + 8,), dtype=tdt, device="cuda")
        res = torch.zeros((E * n,), dtype=tdt, device="cuda")
        imfs = buf[shift:shift + E * M_ * n]
        ws = torch.empty((L.workspace_size(p, [n], E, True),), dtype=torch.uint8, device="cuda")
        L.run(p, xd, [n], 0, E, ws, imfs=imfs, resid_out=res)
        got.append((imfs.clone(), res))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    # one trial at a time through the workspace's own rows: the sum of one is the trial's IMF
    need = L.workspace_size(p, [n], 1, False)
    for small in (False, True):
        for e in range(E):
            s = torch.zeros((M_ * n,), dtype=torch.float64, device="cuda")
            c = torch.zeros((M_,), dtype=torch.int32, device="cuda")
            size = need
            if small:  # the least workspace that is not refused
                lo, hi = 0, need
                while hi - lo > 1:
                    mid = (lo + hi) // 2
                    try:
                        L.run(p, xd[e * n:(e + 1) * n], [n], 0, 1, torch.empty((mid,), dtype=torch.uint8, device="cuda"))
                        hi = mid
                    except L.EngineError as err:
                        assert err.status == L.EEMD_E_NOMEM
                        lo = mid
                size = hi
            ws = torch.empty((size,), dtype=torch.uint8, device="cuda")
            L.run(p, xd[e * n:(e + 1) * n], [n], 0, 1, ws, imf_sum=s, mode_count=c)
            want = got[0][0].view(E, M_, n)[e].double()
            assert torch.equal(s.view(M_, n), want * (c > 0)[:, None])


@pytest.mark.parametrize("E", [1, 7, 8, 9, 17, 300])
def test_ensemble_sum_in_trial_order(E):
    """imf_sum adds the trials that reached a mode in trial order, rounding
    for rounding, whether all did (the first modes) or only some (the last);
    it adds to what the caller's array holds."""
    torch = pytest.importorskip("torch")
    from eemd4cuda_b200 import _lib as L

    n, M_ = 200, 9
    x = torch.from_numpy(rows_of([n], 3)[0]).cuda()
    p = M.make_params(noise_mode=L.EEMD_NOISE_PHILOX, eps=0.5, seed=E, tau=0.25, max_sifts=20, max_imf=M_)
    imfs = torch.zeros((E, M_, n), dtype=torch.float64, device="cuda")
    s = torch.full((M_, n), 0.125, dtype=torch.float64, device="cuda")
    c = torch.full((M_,), 5, dtype=torch.int32, device="cuda")
    nm = torch.zeros((E,), dtype=torch.int32, device="cuda")
    ws = torch.empty((L.workspace_size(p, [n], E, True),), dtype=torch.uint8, device="cuda")
    L.run(p, x, [n], 0, E, ws, imfs=imfs, imf_sum=s, mode_count=c, nmode=nm)
    h, nm = imfs.cpu().numpy(), nm.cpu().numpy()
    for m in range(M_):
        on = [e for e in range(E) if nm[e] > m]
        assert int(c[m]) == 5 + len(on)
        want = np.full(n, 0.125)
        if on:
            acc = h[on[0], m].copy()
            for e in on[1:]:
                acc = acc + h[e, m]
            want = want + acc
        assert np.array_equal(s[m].cpu().numpy(), want), m
    assert E < 300 or len(set(nm)) > 1  # both branches have run


def test_tuned_shapes_give_the_same_imfs():
    """The table's launch shapes for a few short signals (up to 16 CTAs of 512
    samples each) and for an uneven batch against one CTA per task: fixed
    sifts, so the same IMFs bit for bit."""
    torch = pytest.importorskip("torch")
    from eemd4cuda_b200 import _lib as L

    for dtype, lengths, E in [(np.float64, [8192], 1), (np.float32, [3001], 3), (np.float32, [600, 2100, 40000], 4)]:
        rows = rows_of(lengths, 21)
        xd = torch.from_numpy(np.concatenate(rows).astype(dtype)).cuda()
        out = []
        for shape in (None, 1):
            p = M.make_params(dtype=dtype, noise_mode=L.EEMD_NOISE_PHILOX, seed=4, tau=0.0, max_sifts=4, max_imf=3)
            if shape is None:
                p = M.tuned(p, lengths, E)
            else:
                p.cluster_size = 1
            imfs = torch.zeros((3 * E * sum(lengths),), dtype=torch.from_numpy(np.zeros(1, dtype)).dtype, device="cuda")
            ws = torch.empty((L.workspace_size(p, lengths, E, True),), dtype=torch.uint8, device="cuda")
            L.run(p, xd, lengths, 0, E, ws, imfs=imfs)
            out.append(imfs)
        assert torch.equal(out[0], out[1]), lengths
