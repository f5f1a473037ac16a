"""The screened scan of the tensor form (8-bit phenotype bounds, then the exact statistics of
the pairs that pass) against the same library's per-pair dump, which goes through the full
digits: the same hits, F and F2 and the same largest F and F2, bit for bit, at the edges of its
tiles (80 x 42 SNPs), of the packed layouts (128 individuals a stage) and of its range (thresholds
and individuals where it turns to the full digits), over several blocks, traits and masks; and
where the candidate list overflows, since the traits make nearly every pair a hit."""
import numpy as np
import pytest

from epigpu_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _expected(ctx, blocks, t, test, t1, t2):
    """Hits (as a set of rows) and maxima of trait t from the dump of every block."""
    rows, mf, mf2 = set(), -np.inf, -np.inf
    for b, (s1, m1, s2, m2) in enumerate(blocks):
        d = ctx.scan_dump((s1, m1, s2, m2), capi.default_opts(test=test, t1=t1, t2=t2, form=capi.FORM_TENSOR), trait=t)
        tri = (np.arange(m1)[:, None] + s1) > (np.arange(m2)[None, :] + s2)
        F, F2 = d["F"], d["F2"]
        with np.errstate(invalid="ignore"):
            hit = (F > np.float32(t1)) & tri if test == "f" else \
                ((F > np.float32(t1)) | (F2 > np.float32(t2))) & (d["df1"] > 5) & tri
        for i, j in zip(*np.nonzero(hit)):
            rows.add((t, b, i + s1, j + s2, d["df1"][i, j], d["df2"][i, j], F[i, j], F2[i, j] if test == "i" else 0.0))
        ok = tri & ~np.isnan(F)
        if ok.any():
            mf = max(mf, F[ok].max())
        ok = tri & ~np.isnan(F2)
        if test == "i" and ok.any():
            mf2 = max(mf2, F2[ok].max())
    return rows, mf, (mf2 if test == "i" else 0.0)


def _check(ctx, blocks, ntraits, test, t1, t2, tile=0, screened=None):
    opts = capi.default_opts(test=test, t1=t1, t2=t2, form=capi.FORM_TENSOR, report_trait=-1, tile_config=tile)
    hits, total, ex = ctx.scan(blocks, opts, ntraits=ntraits, want_blocks=True, want_traits=True)
    if screened is not None:  # the state reset, the screen and the exact kernel, or the reset and one kernel
        assert (ctx.last_timing()[2] >= 3) == screened
    got = set(zip(ex["trait"], ex["block"], hits["snp1"], hits["snp2"], hits["df1"], hits["df2"], hits["F"], hits["F2"]))
    want = set()
    for t in range(ntraits):
        rows, mf, mf2 = _expected(ctx, blocks, t, test, t1, t2)
        want |= rows
        assert ex["max_f"][t] == np.float32(mf) and ex["max_f2"][t] == np.float32(mf2), t
    assert total == len(hits) == len(got) and got == want
    return total


def _load(ctx, nid, sizes, ntraits, seed, miss=0.01, masks=True):
    nsnp = sum(sizes)
    codes = synth.genotype_codes(nid, nsnp, seed=seed, miss=miss)
    if nsnp > 20:
        codes[3], codes[7], codes[11] = 0, 3, 2   # monomorphic, all missing, monomorphic
    rng = np.random.default_rng(seed + 1)
    pairs = [tuple(rng.choice(nsnp, 2, replace=False)) for _ in range(2)]
    cols = []
    for t in range(ntraits):
        y = synth.planted_phenotype(codes, pairs, seed=seed + 10 + t, var_frac=min(0.3, 60.0 / nid), miss=0.0)
        cols.append(y if t % 2 == 0 else np.exp(y).astype(np.float32))  # every second one skewed
    valid = rng.random((nid, ntraits)) >= (0.03 if masks else 0.0)
    ctx.load_packed(synth.pack(codes), nid)
    ctx.set_traits(np.stack(cols, 1), valid)
    starts = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    return [(int(starts[i]), sizes[i], int(starts[j]), sizes[j]) for i in range(len(sizes)) for j in range(i + 1)]


@pytest.mark.parametrize("nid", [64, 200, 256, 257, 511, 1153])
@pytest.mark.parametrize("sizes", [[2], [42], [43, 80], [81, 85, 1], [167, 121]], ids=str)
@pytest.mark.parametrize("test", ["f", "i"])
def test_tile_edges(gpu_ctx, nid, sizes, test):
    blocks = _load(gpu_ctx, nid, sizes, 2, seed=nid + len(sizes))
    t1, t2 = synth.f_threshold(8, nid - 9, 1e-6), synth.f_threshold(4, nid - 9, 1e-6)
    _check(gpu_ctx, blocks, 2, test, t1, t2, screened=True)


@pytest.mark.parametrize("tile", [1, 2, 3, 4, 5, 6])
def test_variants_and_maxima(gpu_ctx, tile):
    """Every kernel variant with one digit and with two (15,000 individuals); thresholds out of reach, so that the maxima alone drive the screen."""
    for nid, p in ((1500, 1e-5), (15000, 1e-5)):
        blocks = _load(gpu_ctx, nid, [190, 93], 3, seed=5)
        assert _check(gpu_ctx, blocks, 3, "i", synth.f_threshold(8, nid - 9, p), synth.f_threshold(4, nid - 9, p), tile) > 0
        assert _check(gpu_ctx, blocks, 3, "i", 1e6, 1e6, tile) == 0


@pytest.mark.parametrize("ntraits", [4, 5, 8, 13])
@pytest.mark.parametrize("sizes", [[15, 2], [81, 85, 1]], ids=str)
@pytest.mark.parametrize("test", ["f", "i"])
def test_traits_with_one_mask_go_in_groups(gpu_ctx, ntraits, sizes, test):
    """Traits with the same valid individuals, five to a group (a full group and a partial one)."""
    nid = 700
    blocks = _load(gpu_ctx, nid, sizes, ntraits, seed=ntraits, masks=False)
    t1, t2 = synth.f_threshold(8, nid - 9, 1e-5), synth.f_threshold(4, nid - 9, 1e-5)
    _check(gpu_ctx, blocks, ntraits, test, t1, t2, screened=True)
    gpu_ctx.scan(blocks, capi.default_opts(test=test, t1=t1, t2=t2, form=capi.FORM_TENSOR), ntraits=ntraits)
    assert "groups" in gpu_ctx.scan_config()


@pytest.mark.parametrize("nid,screened", [(6017, True), (12200, None), (32641, False)])
def test_many_individuals(gpu_ctx, nid, screened):
    blocks = _load(gpu_ctx, nid, [300, 41], 1, seed=nid, miss=0.02)
    p = 1e-6 if nid < 10000 else 1e-9  # (12,200: two digits)
    _check(gpu_ctx, blocks, 1, "i", synth.f_threshold(8, nid - 9, p), synth.f_threshold(4, nid - 9, p), screened=screened)


def test_thresholds_that_let_many_through_are_not_screened(gpu_ctx):
    blocks = _load(gpu_ctx, 900, [500], 1, seed=77)
    for p, screened in ((1e-2, False), (1e-6, True)):
        _check(gpu_ctx, blocks, 1, "i", synth.f_threshold(8, 891, p), synth.f_threshold(4, 891, p), screened=screened)


def test_candidate_list_overflow():
    """SNPs in strong linkage disequilibrium with a causal one: nearly every pair passes, more than
    the list holds, and the scan is made again with the full digits; the next is not screened."""
    nid, nsnp = 600, 600
    codes = synth.genotype_codes(nid, nsnp, seed=91, miss=0.0)
    rng = np.random.default_rng(92)
    codes = np.where(rng.random((nsnp, nid)) < 0.7, codes[:1], codes).astype(np.uint8)
    y = (codes[0] + 0.5 * rng.standard_normal(nid)).astype(np.float32)
    t1 = synth.f_threshold(8, nid - 9, 1e-6)
    blocks = [(0, nsnp, 0, nsnp)]
    with capi.Context(0) as ctx:  # a new one: its list has the smallest capacity
        ctx.load_packed(synth.pack(codes), nid)
        ctx.set_traits(y)
        total = _check(ctx, blocks, 1, "f", t1, 0.0, screened=False)
        assert total > 1 << 16
        assert _check(ctx, blocks, 1, "f", t1, 0.0, screened=False) == total


@pytest.mark.parametrize("nid", [63, 64, 131, 255])
@pytest.mark.parametrize("test", ["f", "i"])
def test_automatic_form_of_few_individuals(gpu_ctx, nid, test):
    """The automatic choice takes the tensor form from 64 individuals on: the hits of the plain
    form on the same call, with F and F2 within the parity bar (1e-5 SSY / SSW)."""
    blocks = _load(gpu_ctx, nid, [150, 77], 1, seed=nid)
    t1, t2 = synth.f_threshold(8, nid - 9, 1e-4), synth.f_threshold(4, nid - 9, 1e-4)
    opts = dict(test=test, t1=t1, t2=t2)
    auto, n, ex = gpu_ctx.scan(blocks, capi.default_opts(**opts), want_blocks=True)
    assert gpu_ctx.last_timing()[3] == (capi.FORM_TENSOR if nid >= 64 else capi.FORM_POPC)
    plain, m, px = gpu_ctx.scan(blocks, capi.default_opts(form=capi.FORM_POPC, **opts), want_blocks=True)
    assert n == m and np.array_equal(ex["block"], px["block"])
    for f in ("snp1", "snp2", "df1", "df2"):
        assert np.array_equal(auto[f], plain[f])
    kappa = 1.0 + px["max_f"].max() * 8 / (nid - 9)  # the largest SSY / SSW about
    assert np.all(np.abs(auto["F"] - plain["F"]) <= 2e-5 * kappa * np.maximum(plain["F"], 1.0))
    assert np.all(np.abs(auto["F2"] - plain["F2"]) <= 2e-5 * kappa * np.maximum(plain["F2"], 1.0))
    assert np.allclose(ex["max_f"], px["max_f"], rtol=2e-5 * kappa)


@pytest.mark.parametrize("nid", [31, 59, 64, 66, 128, 191, 257])
@pytest.mark.parametrize("miss", [0.0, 0.01, 0.4])
@pytest.mark.parametrize("tile", [1, 2, 3])
def test_plain_form_sums_by_look_up(gpu_ctx, nid, miss, tile):
    """The plain form's cell sums (tables over five individuals, 13 a stage of 64) at the edges of the
    tables, words and stages, without, with few and with many missing calls: the counts and degrees
    of freedom of the tensor form's dump, F and F2 within 1e-5 of SSY in SSB, SSI and SSW."""
    for block in _load(gpu_ctx, nid, [135, 70], 1, seed=nid, miss=miss):
        want = gpu_ctx.scan_dump(block, capi.default_opts(test="i", form=capi.FORM_TENSOR))
        got = gpu_ctx.scan_dump(block, capi.default_opts(test="i", form=capi.FORM_POPC, tile_config=tile))
        s1, m1, s2, m2 = block
        tri = (np.arange(m1)[:, None] + s1) > (np.arange(m2)[None, :] + s2)
        for f in ("counts", "df1", "df2"):
            assert np.array_equal(got[f][tri], want[f][tri])
        ok = tri & (want["df1"] > 0) & (want["df2"] > 2)
        d1, d2 = want["df1"][ok].astype(float), want["df2"][ok].astype(float)
        kappa = 1.0 + want["F"][ok] * d1 / d2  # SSY / SSW
        assert np.all(np.abs(got["F"][ok] - want["F"][ok]) <= 1e-5 * kappa ** 2 * d2 / d1 + 1e-6 * want["F"][ok])
        assert np.all(np.abs(got["F2"][ok] - want["F2"][ok]) <= 1e-5 * kappa ** 2 * d2 / 4 + 1e-6 * want["F2"][ok])


@pytest.mark.parametrize("nid,nsnp,block", [(17, 90, (0, 90, 0, 90)), (128, 130, (0, 130, 0, 130)),
                                            (600, 3100, (0, 3100, 0, 3100)), (1203, 3200, (51, 3090, 3, 3197)),
                                            (2000, 300, (200, 100, 7, 150)), (9001, 201, (0, 201, 0, 201)),
                                            (32700, 50, (0, 50, 0, 50))], ids=str)
@pytest.mark.parametrize("test", ["f", "i"])
def test_block_scan_without_allocation(gpu_ctx, nid, nsnp, block, test):
    """epi_scan_block_noalloc builds the operands from the packed words (a full or a partial last
    one) and goes through a block in parts of 3,072 SNPs: the rows and maxima of epi_scan, bit for
    bit where both go by the digits, within the parity bar where the plain kernel runs (32,700)."""
    import ctypes
    torch = pytest.importorskip("torch")
    codes = synth.genotype_codes(nid, nsnp, seed=nid)
    codes[3], codes[7], codes[11] = 0, 3, 2
    y = synth.planted_phenotype(codes, [(1, 20), (33, 5)], seed=nid, var_frac=min(0.3, 60.0 / nid), miss=0.02)
    packed = synth.pack(codes)
    t1, t2 = synth.f_threshold(8, max(nid - 9, 2), 1e-5), synth.f_threshold(4, max(nid - 9, 2), 1e-5)
    opts = capi.default_opts(test=test, t1=t1, t2=t2, form=capi.FORM_TENSOR)
    gpu_ctx.load_packed(packed, nid)
    gpu_ctx.set_phenotype(y)
    want, n, ex = gpu_ctx.scan([block], opts)
    want = want[np.lexsort((want["snp2"], want["snp1"]))]
    gp, ph = torch.from_numpy(packed).cuda(), torch.from_numpy(y).cuda()
    rows = torch.zeros((1 << 16, 6), dtype=torch.int32, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    maxf = torch.zeros(2, dtype=torch.float32, device="cuda")
    b = capi.Block(*block)
    for _ in range(2):
        st = capi.load().epi_scan_block_noalloc(gp.data_ptr(), nid, nsnp, ph.data_ptr(), ctypes.byref(b),
                                                ctypes.byref(opts), rows.data_ptr(), rows.shape[0],
                                                count.data_ptr(), maxf.data_ptr(), None)
        assert st == capi.EPI_OK and int(count) == n
        got = rows[:n].cpu().numpy().copy().view(capi.HIT_DTYPE).reshape(-1)
        got = got[np.lexsort((got["snp2"], got["snp1"]))]
        top = np.array([ex["max_f"][0], ex["max_f2"][0]])
        if nid <= 2000:  # (above, too many pairs pass the screen at these thresholds: the plain kernel)
            assert np.array_equal(got, want) and np.array_equal(maxf.cpu().numpy(), top)
        else:
            assert all(np.array_equal(got[f], want[f]) for f in ("snp1", "snp2", "df1", "df2"))
            assert np.allclose(got["F"], want["F"], rtol=2e-5) and np.allclose(maxf.cpu().numpy(), top, rtol=2e-5)
