"""What the screens may settle: their bounds of F and F2 against the same library's per-pair dump
(which goes through no screen) and, at a small size, against the FP64 oracle, on data that press
the bounds -- maxima unknown to many warps at once, traits whose sum of squares sits in a few
individuals that a pair misses, SNPs with hardly a call, pairs that explain nothing at all."""
import numpy as np
import pytest

from epigpu_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _dumped(ctx, block, test, form, trait=0, **opts):
    """F, F2 and df1 of the block's pairs snp1 > snp2, and those pairs."""
    d = ctx.scan_dump(block, capi.default_opts(test=test, form=form, **opts), trait=trait)
    s1, m1, s2, m2 = block
    i, j = np.nonzero((np.arange(m1)[:, None] + s1) > (np.arange(m2)[None, :] + s2))
    return d["F"][i, j], d["F2"][i, j], d["df1"][i, j], i + s1, j + s2


def _maxima(F, F2, test):
    return np.float32(np.nanmax(F)), np.float32(np.nanmax(F2) if test == "i" else 0.0)


@pytest.mark.parametrize("masks", [False, True], ids=["one mask", "own masks"])
def test_unknown_maxima_of_many_traits(gpu_ctx, masks):
    """64 traits, thresholds out of reach: every trait's first units begin without a lower bound of
    its maxima, in every cluster at once, while others raise it."""
    nid, nsnp, ntraits = 700, 330, 64
    rng = np.random.default_rng(3)
    codes = synth.genotype_codes(nid, nsnp, seed=4, miss=0.01)
    y = rng.standard_normal((nid, ntraits)).astype(np.float32)
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_traits(y, rng.random((nid, ntraits)) >= 0.05 if masks else None)
    block = (0, nsnp, 0, nsnp)
    for _ in range(3):
        _, total, ex = gpu_ctx.scan([block], capi.default_opts(test="i", t1=1e6, t2=1e6), ntraits=ntraits)
        assert total == 0 and "screen" in gpu_ctx.scan_config()
        for t in range(0, ntraits, 9):
            F, F2, *_ = _dumped(gpu_ctx, block, "i", capi.FORM_TENSOR, trait=t)
            assert (ex["max_f"][t], ex["max_f2"][t]) == _maxima(F, F2, "i"), t


def _check_thresholds(ctx, block, test, form, among, seed, n=24, config=None):
    """Thresholds a relative 1e-4 below F of pairs drawn from `among` (a mask of the dumped pairs): each scan
    must return that pair and all others above, and the dump's maxima."""
    F, F2, df1, i, j = _dumped(ctx, block, test, form)
    top = np.flatnonzero(among & (F > 0))
    top = top[np.argsort(F[top])[-400:]]
    for k in np.random.default_rng(seed).choice(top, n, replace=False):
        t1 = np.float32(F[k] * np.float32(1.0 - 1e-4))
        hits, total, ex = ctx.scan([block], capi.default_opts(test=test, form=form, t1=t1, t2=1e30))
        if config is not None:
            assert config in ctx.scan_config()
        want = (F > t1) & ((df1 > 5) if test == "i" else True)
        got = set(zip(hits["snp1"], hits["snp2"], hits["F"]))
        assert total == want.sum() and got == set(zip(i[want], j[want], F[want]))
        assert (ex["max_f"][0], ex["max_f2"][0]) == _maxima(F, F2, test)


@pytest.mark.parametrize("test", ["f", "i"])
@pytest.mark.parametrize("nid,sd", [(1000, 3e3), (1000, 1e4), (4000, 3e4)])
def test_plain_form_with_outliers_that_pairs_miss(gpu_ctx, nid, sd, test):
    """Two opposite outliers hold nearly all of the trait's sum of squares; a pair that misses one at
    either SNP keeps a millionth of it and less. No hit and no maximum may be lost."""
    nsnp = 240
    codes = synth.genotype_codes(nid, nsnp, seed=nid, miss=0.0)
    codes[:nsnp // 2, 0], codes[nsnp // 2:, 1] = 3, 3
    y = np.random.default_rng(nid + 1).standard_normal(nid)
    y[0], y[1] = sd, -sd
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_phenotype(y.astype(np.float32))
    block = (0, nsnp, 0, nsnp)
    *_, i, j = _dumped(gpu_ctx, block, test, capi.FORM_POPC)
    _check_thresholds(gpu_ctx, block, test, capi.FORM_POPC, (i >= nsnp // 2) & (j < nsnp // 2), 5)


@pytest.mark.parametrize("miss", [0.4, 0.97])
@pytest.mark.parametrize("test", ["f", "i"])
def test_plain_form_with_many_missing_calls(gpu_ctx, miss, test):
    nid, nsnp = 1500, 200
    codes = synth.genotype_codes(nid, nsnp, seed=17, miss=0.0)
    codes[nsnp // 2:][np.random.default_rng(18).random((nsnp - nsnp // 2, nid)) < miss] = 3
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_phenotype(np.random.default_rng(19).standard_normal(nid).astype(np.float32))
    block = (0, nsnp, 0, nsnp)
    *_, i, j = _dumped(gpu_ctx, block, test, capi.FORM_POPC)
    _check_thresholds(gpu_ctx, block, test, capi.FORM_POPC, (i >= nsnp // 2) & (j < nsnp // 2), 6)


@pytest.mark.parametrize("nid,ntraits,config", [(30700, 1, "8-bit screen"), (30700, 4, "groups"), (15000, 1, "16-bit screen")])
def test_screen_with_snps_of_a_dozen_calls(gpu_ctx, nid, ntraits, config):
    """SNPs known in a dozen individuals against SNPs known in all, where the screen's phenotype is exact
    (two values) or nearly (16 bits): a pair's sum of squares is a difference of floats thousands of
    times its size, and E widens the bounds by next to nothing. (The counts of the two values, 15,271 of
    30,700 and 6 of 12, leave Q 2.4e-4 too large.)"""
    sparse, full, calls = 150, 210, 12
    codes = synth.genotype_codes(nid, sparse + full, seed=nid, miss=0.0)
    rng = np.random.default_rng(nid + 1)
    y = rng.standard_normal(nid)
    high = y >= np.sort(y)[-15271] if nid == 30700 else y >= 0
    if nid == 30700:
        y = np.where(high, 1.0, -1.0)
    for s in range(sparse):
        keep = np.concatenate([rng.choice(np.flatnonzero(high == h), calls // 2, replace=False) for h in (True, False)])
        gone = np.ones(nid, dtype=bool)
        gone[keep] = False
        codes[s, gone] = 3
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_traits(np.repeat(y[:, None], ntraits, 1).astype(np.float32))
    block = (0, sparse + full, 0, sparse + full)
    F, F2, df1, i, j = _dumped(gpu_ctx, block, "f", capi.FORM_TENSOR)
    values = np.unique(F[(j < sparse) & (i >= sparse) & np.isfinite(F) & (F > 3) & (F < 1e5)])
    assert len(values) >= 5
    for v in values[-24:]:
        t1 = np.float32(v * np.float32(1.0 - 1e-4))
        hits, total, ex = gpu_ctx.scan([block], capi.default_opts(t1=t1, form=capi.FORM_TENSOR), ntraits=ntraits)
        assert config in gpu_ctx.scan_config()
        want = F > t1
        assert total == want.sum() and set(zip(hits["snp1"], hits["snp2"])) == set(zip(i[want], j[want]))
        assert ex["max_f"][0] == _maxima(F, F2, "f")[0]


def _noalloc(packed, nid, y, block, **opts):
    """epi_scan_block_noalloc on copies of the inputs: status, rows, maxima of F and F2."""
    torch = pytest.importorskip("torch")
    import ctypes
    gp, ph = torch.from_numpy(packed).cuda(), torch.from_numpy(np.ascontiguousarray(y, dtype=np.float32)).cuda()
    rows = torch.zeros((1 << 20, 6), dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    maxf = torch.zeros(2, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    o, b = capi.default_opts(**opts), capi.Block(*block)
    st = capi.load().epi_scan_block_noalloc(gp.data_ptr(), nid, packed.shape[0], ph.data_ptr(), ctypes.byref(b),
                                            ctypes.byref(o), rows.data_ptr(), rows.shape[0], count.data_ptr(),
                                            maxf.data_ptr(), None)
    got = rows[:int(count)].cpu().numpy().copy().view(capi.HIT_DTYPE).reshape(-1)
    return st, got[np.lexsort((got["snp2"], got["snp1"]))], maxf.cpu().numpy()


@pytest.mark.parametrize("test", ["f", "i"])
@pytest.mark.parametrize("ntraits", [1, 4])
@pytest.mark.parametrize("nid", [256, 1024])
def test_pairs_that_explain_nothing(gpu_ctx, nid, ntraits, test):
    """Two halves with the same genotypes and opposite values of +-1: every cell's sum is 0, the screen's
    phenotype is exact and every F is 0. The largest is 0, not the -inf of no pair."""
    nsnp = 100
    codes = np.tile(synth.genotype_codes(nid // 2, nsnp, seed=nid, miss=0.01), 2)
    half = np.where(np.random.default_rng(1).random((nid // 2, ntraits)) < 0.5, 1.0, -1.0)
    y = np.concatenate([half, -half]).astype(np.float32)
    packed, block = synth.pack(codes), (0, nsnp, 0, nsnp)
    gpu_ctx.load_packed(packed, nid)
    gpu_ctx.set_traits(y)
    for t1 in (0.0, 5.0):
        _, total, ex = gpu_ctx.scan([block], capi.default_opts(test=test, t1=t1, t2=t1, form=capi.FORM_TENSOR),
                                    ntraits=ntraits)
        F, F2, *_ = _dumped(gpu_ctx, block, test, capi.FORM_TENSOR)
        assert total == 0 and _maxima(F, F2, test) == (0.0, 0.0)
        assert np.all(ex["max_f"] == 0.0) and np.all(ex["max_f2"] == 0.0)
    st, rows, top = _noalloc(packed, nid, y[:, 0], block, test=test, t1=5.0, t2=5.0)
    assert st == capi.EPI_OK and len(rows) == 0 and np.array_equal(top, [0.0, 0.0])


@pytest.mark.parametrize("form", [capi.FORM_POPC, capi.FORM_TENSOR], ids=["plain", "tensor"])
def test_dump_of_one_output(gpu_ctx, form):
    """Every output of epi_scan_dump by itself, the others null."""
    import ctypes
    nid, nsnp = 300, 60
    codes = synth.genotype_codes(nid, nsnp, seed=8)
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_phenotype(synth.phenotype(nid, seed=9))
    block = (0, nsnp, 0, nsnp)
    o, b = capi.default_opts(test="i", form=form), capi.Block(*block)
    whole = gpu_ctx.scan_dump(block, o)
    for k, name in enumerate(("counts", "F", "F2", "df1", "df2")):
        out = np.full_like(whole[name], -77)
        args = [None] * 5
        args[k] = out.ctypes.data_as(ctypes.c_void_p)
        assert gpu_ctx.lib.epi_scan_dump(gpu_ctx.h, ctypes.byref(b), ctypes.byref(o), 0, *args) == capi.EPI_OK
        i, j = np.tril_indices(nsnp, -1)
        np.testing.assert_array_equal(out[i, j], whole[name][i, j], err_msg=name)
        assert np.all(out[j, i] == -77)  # pairs that are not tested are left alone


def test_more_segments_than_counters(gpu_ctx):
    """Two traits of 100,000 SNPs at 8,000 individuals and p = 4e-5: more than eight segments, so their
    candidate counters come round again. The same hits and maxima as from 15 scans of eight segments at most."""
    nid, nsnp, ntraits = 8000, 100000, 2
    rng = np.random.default_rng(31)
    gpu_ctx.load_packed(synth.packed_on_gpu(nid, nsnp, seed=32), nid)
    gpu_ctx.set_traits(rng.standard_normal((nid, ntraits)).astype(np.float32), rng.random((nid, ntraits)) >= 0.02)
    opts = capi.default_opts(test="i", t1=synth.f_threshold(8, nid - 9, 4e-5), t2=synth.f_threshold(4, nid - 9, 4e-5),
                             report_trait=-1)

    def scan(block):
        hits, total, ex = gpu_ctx.scan([block], opts, ntraits=ntraits, want_traits=True)
        assert "8-bit screen" in gpu_ctx.scan_config() and total == len(hits) > 0
        return hits, ex["trait"], ex["max_f"], ex["max_f2"], gpu_ctx.last_timing()[2]

    def ordered(hits, trait):
        o = np.lexsort((hits["snp2"], hits["snp1"], trait))
        return hits[o], trait[o]
    hits, trait, mf, mf2, launches = scan((0, nsnp, 0, nsnp))
    assert launches > 1 + 2 * 8
    parts = [scan((i, 20000, j, 20000)) for i in range(0, nsnp, 20000) for j in range(0, i + 1, 20000)]
    assert max(p[4] for p in parts) <= 1 + 2 * 8
    for a, b in zip(ordered(hits, trait), ordered(np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))):
        assert np.array_equal(a, b)
    assert np.array_equal(np.max([p[2] for p in parts], 0), mf) and np.array_equal(np.max([p[3] for p in parts], 0), mf2)


@pytest.mark.parametrize("nid,nsnp,p,test", [(10000, 3300, 1e-6, "i"), (9500, 3000, 1e-6, "f"), (8000, 3000, 1e-6, "f")])
def test_block_scan_in_parts_that_its_list_holds(gpu_ctx, nid, nsnp, p, test):
    """epi_scan_block_noalloc where a part of 3,072 SNPs a side passes on more pairs than its list holds (no
    effects, so the largest F is near): the second pass's small first part holds them, so the rows are the
    exact kernel's, those of epi_scan bit for bit, and not the plain kernel's."""
    codes = synth.genotype_codes(nid, nsnp, seed=nid, miss=0.01)
    y = synth.phenotype(nid, seed=nid)
    packed, block = synth.pack(codes), (0, nsnp, 0, nsnp)
    opts = dict(test=test, t1=synth.f_threshold(8, nid - 9, p), t2=synth.f_threshold(4, nid - 9, p))
    gpu_ctx.load_packed(packed, nid)
    gpu_ctx.set_phenotype(y)
    want, n, ex = gpu_ctx.scan([block], capi.default_opts(form=capi.FORM_TENSOR, **opts))
    want = want[np.lexsort((want["snp2"], want["snp1"]))]
    st, rows, top = _noalloc(packed, nid, y, block, **opts)
    assert st == capi.EPI_OK and n > 0 and np.array_equal(rows, want)
    assert np.array_equal(top, [ex["max_f"][0], ex["max_f2"][0]])


@pytest.mark.parametrize("test", ["f", "i"])
@pytest.mark.parametrize("where", ["first part", "last part"])
def test_block_scan_whose_list_runs_over(gpu_ctx, where, test):
    """SNPs in linkage around a strong effect fill the list of one part, the first or the last of four, which
    have given rows, a count and maxima by then: all of it is made again by the plain kernel."""
    nid, nsnp, linked = 600, 3500, 150
    codes = synth.genotype_codes(nid, nsnp, seed=41, miss=0.01)
    rng = np.random.default_rng(42)
    at = 0 if where == "first part" else nsnp - linked
    keep = rng.random((linked, nid)) < 0.85
    codes[at:at + linked] = np.where(keep, codes[at], codes[at:at + linked])
    pairs = [(5, 3), (900, 200), (3000, 1500)] if at else [(nsnp - 3, nsnp - 9), (2000, 1900), (3400, 800)]
    y = synth.planted_phenotype(codes, pairs, seed=43, var_frac=0.08, miss=0.01)
    y = np.where(y == -9.0, y, y + 0.8 * np.where(codes[at] == 3, 0, codes[at])).astype(np.float32)
    packed, block = synth.pack(codes), (0, nsnp, 0, nsnp)
    opts = dict(test=test, t1=synth.f_threshold(8, nid - 9, 1e-6), t2=synth.f_threshold(4, nid - 9, 1e-6))
    gpu_ctx.load_packed(packed, nid)
    gpu_ctx.set_phenotype(y)
    want, n, ex = gpu_ctx.scan([block], capi.default_opts(form=capi.FORM_TENSOR, **opts))
    want = want[np.lexsort((want["snp2"], want["snp1"]))]
    assert n > 8000 + len(pairs)
    for _ in range(2):
        st, rows, top = _noalloc(packed, nid, y, block, **opts)
        assert st == capi.EPI_OK
        # (F of the plain kernel's FP32 sums: a pair at a threshold may fall on its other side)
        both = {(a, b): f for a, b, f in zip(want["snp1"], want["snp2"], want["F"])}
        got = {(a, b): f for a, b, f in zip(rows["snp1"], rows["snp2"], rows["F"])}
        assert len(got) == len(rows) and abs(len(rows) - n) <= 3 and len(both.keys() ^ got.keys()) <= 3
        common = sorted(both.keys() & got.keys())
        np.testing.assert_allclose([got[k] for k in common], [both[k] for k in common], rtol=2e-5)
        assert not np.array_equal([got[k] for k in common], [both[k] for k in common])  # the plain kernel's
        np.testing.assert_allclose(top, [ex["max_f"][0], ex["max_f2"][0]], rtol=2e-5)


@pytest.mark.parametrize("nid", [64, 101, 150, 255])
@pytest.mark.parametrize("sd", [0.0, 1e3], ids=["normal", "outlier"])
@pytest.mark.parametrize("test", ["f", "i"])
def test_few_individuals_keep_32_bits(gpu_ctx, nid, sd, test):
    """The automatic form of 64 to 255 individuals evaluates from the phenotype in 32 bits, as the plain form
    does: F and F2 of every pair against FP64, with an outlier that most pairs miss (24-bit fixed point is
    good to 2^-24 of the outlier). y carries a relative 2^-24, which moves the roots of SSB, SSI and SSW by
    2^-24 of the norm of y over the pair's individuals; F is rounded to 32 bits."""
    nsnp, u = 31, 2.0 ** -24
    codes = synth.genotype_codes(nid, nsnp, seed=nid, miss=0.02)
    codes[4:, 0] = 3
    y = np.random.default_rng(nid).standard_normal(nid).astype(np.float32)
    if sd:
        y[0] = sd
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_phenotype(y)
    hits, total, ex = gpu_ctx.scan([(0, nsnp, 0, nsnp)], capi.default_opts(test=test, safe=1, t1=1e-3, t2=1e-3))
    assert "screen" in gpu_ctx.scan_config() and total > nsnp * (nsnp - 1) // 2 - 60
    yc = y.astype(np.float64) - y.astype(np.float64).mean()
    for h in hits:
        gi, gj = codes[h["snp1"]], codes[h["snp2"]]
        ok = (gi != 3) & (gj != 3)
        cell, v = 3 * gi[ok].astype(int) + gj[ok], yc[ok]
        n, S = np.bincount(cell, minlength=9), np.bincount(cell, v, minlength=9)
        m, mc = v.mean(), S / np.maximum(n, 1)
        ssb, ssw, d1, d2 = (n * (mc - m) ** 2).sum(), ((v - mc[cell]) ** 2).sum(), (n > 0).sum() - 1, ok.sum() - (n > 0).sum()
        assert (h["df1"], h["df2"]) == (d1, d2)
        norm = np.sqrt((v ** 2).sum())

        def near(got, ss, df):
            want = ss / df / (ssw / d2)
            tol = u * (1.0 + 2.2 * norm / np.sqrt(ss) + 2.2 * norm / np.sqrt(ssw))
            assert abs(got - want) <= tol * want, (got, want, tol)
        near(h["F"], ssb, d1)
        if test == "i":
            n3, S3 = n.reshape(3, 3), S.reshape(3, 3)
            row, col = S3.sum(1) / np.maximum(n3.sum(1), 1), S3.sum(0) / np.maximum(n3.sum(0), 1)
            near(h["F2"], (n3 * (mc.reshape(3, 3) - row[:, None] - col[None] + m) ** 2).sum(), 4)
    assert ex["max_f"][0] == hits["F"].max()


def test_block_scan_without_allocation_times_out(gpu_ctx):
    """A wait of the screen that runs out after wait_limit_ms ends epi_scan_block_noalloc with a status; the
    next call is whole."""
    import time
    nid, nsnp = 1203, 300
    codes = synth.genotype_codes(nid, nsnp, seed=61)
    packed, y, block = synth.pack(codes), synth.phenotype(nid, seed=62), (0, nsnp, 0, nsnp)
    opts = dict(test="i", t1=synth.f_threshold(8, nid - 9, 1e-3), t2=synth.f_threshold(4, nid - 9, 1e-3))
    st, want, top = _noalloc(packed, nid, y, block, **opts)
    assert st == capi.EPI_OK and len(want) > 0
    t = time.perf_counter()
    st, *_ = _noalloc(packed, nid, y, block, wait_limit_ms=20, debug=capi.DEBUG_STALL, **opts)
    assert st == capi.EPI_E_TIMEOUT and time.perf_counter() - t < 10.0
    for limit in (0, 20, -1):
        st, rows, again = _noalloc(packed, nid, y, block, wait_limit_ms=limit, **opts)
        assert st == capi.EPI_OK and np.array_equal(rows, want) and np.array_equal(again, top)


@pytest.mark.parametrize("nid,nsnp,ntraits,form,config",
                         [(96, 150, 1, capi.FORM_AUTO, "8-bit screen"), (96, 150, 1, capi.FORM_TENSOR, "8-bit screen"),
                          (300, 167, 1, capi.FORM_AUTO, "8-bit screen"), (1153, 200, 1, capi.FORM_AUTO, "8-bit screen"),
                          (700, 130, 5, capi.FORM_AUTO, "groups"), (15000, 140, 1, capi.FORM_AUTO, "16-bit screen")])
@pytest.mark.parametrize("test", ["f", "i"])
def test_screened_scans_against_the_oracle(gpu_ctx, nid, nsnp, ntraits, form, config, test):
    """The screen and the exact kernel against the FP64 oracle: the hits in its order, F within the parity bar
    and the largest F, for every trait that is asked for in turn."""
    import oracles
    import parity
    codes = synth.genotype_codes(nid, nsnp, seed=nid, miss=0.01)
    block = (0, nsnp, 0, nsnp)
    cols = np.stack([synth.planted_phenotype(codes, [(1, 20), (33, 5)], seed=nid + t, var_frac=min(0.3, 60.0 / nid), miss=0.0)
                     for t in range(ntraits)], 1)
    gpu_ctx.load_packed(synth.pack(codes), nid)
    gpu_ctx.set_traits(cols, np.ones(cols.shape, dtype=np.uint8))
    p = 1e-4 if nid < 15000 else 1e-3
    t1, t2 = synth.f_threshold(8, nid - 9, p), synth.f_threshold(4, nid - 9, p)
    for t in range(ntraits):
        want, _, per = oracles.oracle_scan_block(codes, cols[:, t], block, test=test, t1=t1, t2=t2, per_pair=True)
        near = parity.near_threshold(per, block, t1, t2, test, 1e-4)
        opts = capi.default_opts(test=test, t1=t1, t2=t2, form=form, report_trait=t)
        hits, total, ex = gpu_ctx.scan([block], opts, ntraits=ntraits)
        assert config in gpu_ctx.scan_config() and total == len(hits) > 0
        ok, msg = parity.compare_hit_lists(hits, want, near)
        assert ok, msg
        assert parity.f_errors(hits, per, block, 1e-5).max() <= 1.0
        F = np.where(per["df1"] > 0, per["F"], -np.inf)[np.tril_indices(nsnp, -1)]
        k = np.nanmax(F) * 8.0 / (nid - 9)  # about the largest SSB / SSW
        assert abs(ex["max_f"][t] - np.nanmax(F)) <= 1e-5 * (1.0 + k) * np.nanmax(F)


@pytest.mark.parametrize("nid", [150, 400, 3000])
@pytest.mark.parametrize("test", ["f", "i"])
def test_pairs_of_individuals_with_one_value(gpu_ctx, nid, test):
    """SNPs known in a few individuals who all have the same value of a trait of two or three: nothing is
    there to explain, F is 0/0 and not the infinity of a rounding over nothing. No hit, no maximum, in the
    automatic form, the tensor form and the allocation-free call."""
    nsnp, sparse = 90, 30
    codes = synth.genotype_codes(nid, nsnp, seed=nid, miss=0.0)
    rng = np.random.default_rng(nid + 1)
    y = rng.integers(0, 3 if nid == 400 else 2, nid).astype(np.float32)
    for s in range(sparse):
        gone = np.ones(nid, dtype=bool)
        gone[rng.choice(np.flatnonzero(y == s % 2), 5 + s % 7, replace=False)] = False
        codes[s, gone] = 3
    packed, block = synth.pack(codes), (0, nsnp, 0, nsnp)
    t1, t2 = synth.f_threshold(8, nid - 9, 1e-3), synth.f_threshold(4, nid - 9, 1e-3)
    gpu_ctx.load_packed(packed, nid)
    gpu_ctx.set_phenotype(y)
    F, F2, df1, i, j = _dumped(gpu_ctx, block, test, capi.FORM_TENSOR)
    flat = j < sparse
    top = np.nanmax(F[~flat])
    for form in (capi.FORM_AUTO, capi.FORM_TENSOR):
        hits, _, ex = gpu_ctx.scan([block], capi.default_opts(test=test, safe=1, t1=t1, t2=t2, form=form))
        assert np.all(hits["snp2"] >= sparse) and abs(ex["max_f"][0] - top) <= 2e-5 * top
    st, rows, most = _noalloc(packed, nid, y, block, test=test, safe=1, t1=t1, t2=t2)
    assert st == capi.EPI_OK and np.all(rows["snp2"] >= sparse) and abs(most[0] - top) <= 2e-5 * top
    assert not np.any(F[flat] > 0.01) and not (test == "i" and np.any(F2[flat] > 0.01))
