"""The library's host side (epi_capi.cu) over a CUDA runtime and kernels that do nothing
(fake/fake_cuda.cpp): what a context holds after an allocation has failed, and which kernels a
scan is given. No GPU: the fake checks that every launch's memory is allocated."""
import ctypes
import pathlib
import subprocess

import numpy as np
import pytest

from epigpu_b200 import build, capi, synth

HERE = pathlib.Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    nvcc, inc = build._nvcc(), ["-I", str(build.INCLUDE), "-I", str(build.CSRC)]
    capi_o, fake_o, so = (str(d / n) for n in ("capi.o", "fake.o", "libfake.so"))
    flags = [f for f in build.NVCC_FLAGS if f != "-lineinfo"]
    subprocess.run([nvcc, *flags, *inc, "-c", str(build.CSRC / "epi_capi.cu"), "-o", capi_o], check=True)
    subprocess.run([nvcc, *flags, *inc, "-c", str(HERE / "fake" / "fake_cuda.cpp"), "-o", fake_o], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", capi_o, fake_o, "-o", so, "-lpthread"], check=True)
    syms = subprocess.run(["nm", "-D", "--undefined-only", so], capture_output=True, text=True).stdout
    assert "cuda" not in syms, syms  # nothing left to a real runtime
    # (the allocation-free call is in another file of the library)
    sigs = dict(capi._SIGS)
    del sigs["epi_scan_block_noalloc"]
    lib = ctypes.CDLL(so)
    for name, (res, args) in sigs.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.fake_error.restype = ctypes.c_char_p
    lib.fake_limit.argtypes = [ctypes.c_size_t]
    lib.fake_used.restype = ctypes.c_size_t
    lib.fake_rate.argtypes = [ctypes.c_double]
    lib.fake_traits.argtypes = [ctypes.c_double] * 3
    return lib


class Ctx:
    """A context over the fake runtime; every call is checked for launches on memory that is not there."""

    def __init__(self, lib):
        self.lib, self.h = lib, ctypes.c_void_p()
        lib.fake_reset()
        assert lib.epi_open(0, ctypes.byref(self.h)) == capi.EPI_OK
        self.nid = self.nsnp = self.ntraits = 0

    def _done(self, st):
        assert self.lib.fake_error() == b"", self.lib.fake_error()
        return st

    def load(self, nid, nsnp):
        g = np.zeros((nsnp, (nid + 15) // 16), dtype=np.int32)
        self.nid, self.nsnp = nid, nsnp
        return self._done(self.lib.epi_load_packed(self.h, g.ctypes.data, nid, nsnp, nid // 16, nid % 16))

    def traits(self, ntraits=1):
        y = np.zeros((ntraits, self.nid), dtype=np.float32)
        self.ntraits = ntraits
        return self._done(self.lib.epi_set_traits(self.h, y.ctypes.data, self.nid, ntraits, None))

    def scan(self, blocks=None, **opts):
        """Status, and the launches by kind: the kernel with all digits and with the screens 1 to 3, the
        exact kernel, the plain kernel; and the graphs captured."""
        o = capi.default_opts(**opts)
        arr = capi.blocks_array(blocks or [(0, self.nsnp, 0, self.nsnp)])
        n = (ctypes.c_int * 7)()
        self.lib.fake_count(n)
        nh = ctypes.c_int64()
        st = self.lib.epi_scan(self.h, ctypes.cast(arr, ctypes.c_void_p), len(blocks or [0]), ctypes.byref(o), None, 0,
                               ctypes.byref(nh), None, None, None, None)
        self.lib.fake_count(n)
        names = ("full", "one", "two", "groups", "exact", "plain", "captures")
        return self._done(st), {k: v for k, v in zip(names, n) if v}

    def close(self):
        self.lib.epi_close(self.h)
        assert self.lib.fake_error() == b"" and self.lib.fake_used() == 0  # all memory given back


@pytest.fixture
def ctx(library):
    c = Ctx(library)
    yield c
    c.close()


HIGH, LOW = dict(t1=8.0, t2=11.0), dict(t1=0.5, t2=0.5)  # screened, and not (one pair in 400 or more passes)
STREAMED = dict(form=capi.FORM_TENSOR, tile_config=6)


@pytest.mark.parametrize("first,second", [(HIGH, LOW), (LOW, HIGH)], ids=["one digit, all", "all, one digit"])
def test_expanded_rows_after_a_failed_allocation(ctx, first, second):
    """A scan that changes the kind of expanded rows frees the old ones; where the new ones then cannot
    be allocated, the next scan of the first kind has to expand its rows again."""
    assert ctx.load(4000, 100000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    for failing in range(4):
        assert ctx.scan(**STREAMED, **first)[0] == capi.EPI_OK
        ctx.lib.fake_fail_after(failing)
        ctx.scan(**STREAMED, **second)
        ctx.lib.fake_fail_after(-1)
        assert ctx.scan(**STREAMED, **first)[0] == capi.EPI_OK


@pytest.mark.parametrize("form", [capi.FORM_TENSOR, capi.FORM_POPC], ids=["tensor", "plain"])
def test_a_load_that_fails_leaves_no_genotypes(ctx, form):
    """Whichever allocation of a larger upload fails, the next scan is refused; the context is whole again
    after the next upload, its traits kept where the number of individuals is the same."""
    for failing in range(8):
        assert ctx.load(1000, 300) == capi.EPI_OK and ctx.traits(2) == capi.EPI_OK
        assert ctx.scan(form=form, **HIGH)[0] == capi.EPI_OK
        ctx.lib.fake_fail_after(failing)
        st = ctx.load(1000, 400 * (failing + 1))
        ctx.lib.fake_fail_after(-1)
        if st != capi.EPI_OK:
            assert st == capi.EPI_E_NOMEM
            assert ctx.scan(form=form, **HIGH) == (capi.EPI_E_STATE, {})
            assert ctx.load(1000, 300) == capi.EPI_OK
        assert ctx.scan(form=form, **HIGH)[0] == capi.EPI_OK


def test_traits_and_scans_that_fail_leave_nothing_half_done(ctx):
    """Every allocation of a larger set of traits and of the scan after it fails once; the calls after
    that, with these or with fewer traits, find memory for all that they launch."""
    assert ctx.load(1000, 300) == capi.EPI_OK
    for form in (capi.FORM_TENSOR, capi.FORM_POPC):
        for failing in range(16):
            assert ctx.traits(1) == capi.EPI_OK and ctx.scan(form=form, **HIGH)[0] == capi.EPI_OK
            ctx.lib.fake_fail_after(failing)
            ctx.nsnp = 300
            if ctx.traits(40 * (failing + 1)) == capi.EPI_OK:
                ctx.scan(form=form, **HIGH)
            else:
                assert ctx.scan(form=form, **HIGH)[0] == capi.EPI_E_STATE
            ctx.lib.fake_fail_after(-1)
            assert ctx.traits(3) == capi.EPI_OK and ctx.scan(form=form, **HIGH)[0] == capi.EPI_OK


def test_expanded_rows_make_room_for_a_larger_fileset(ctx):
    """The rows of the fileset before it (20 GB) are given back where the new one does not fit beside them."""
    assert ctx.load(4000, 800000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    assert ctx.scan(**STREAMED, **HIGH)[0] == capi.EPI_OK
    used = ctx.lib.fake_used()
    assert used > 35e9
    ctx.lib.fake_limit(used + (4 << 30))
    assert ctx.load(4000, 1600000) == capi.EPI_OK
    ctx.lib.fake_limit(180 << 30)
    assert ctx.scan(**STREAMED, **HIGH)[0] == capi.EPI_OK


@pytest.mark.parametrize("free_mb", list(range(34, 100, 8)) + list(range(100, 700, 50)))
def test_a_scan_that_the_screen_has_no_room_for(ctx, free_mb):
    """The hits' buffer (32 MB) is all that a first scan cannot do without: where the candidates' list or
    the expanded rows (100 and 184 MB here) do not fit, the kernel with all digits makes the scan."""
    assert ctx.load(1000, 30000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    ctx.lib.fake_limit(ctx.lib.fake_used() + (free_mb << 20))
    for _ in range(2):
        st, n = ctx.scan(**HIGH)
        assert st == capi.EPI_OK and (n.get("one", 0) > 0 or n.get("full", 0) > 0)
    if free_mb >= 650:
        assert n == {"one": 1, "exact": 1}


def _share(t1, t2, test, nid, pairs, r):
    """The share of a trait's pairs that the screen is expected to pass on (epi_capi.cu: screen_share)."""
    from scipy import stats
    total = 0.0
    for df, thr in ((8, t1), (4, t2))[:2 if test == "i" else 1]:
        top = np.sqrt(stats.chi2.isf(1.0 / pairs, df))
        root = min(top - r, np.sqrt(df * thr * nid / (nid - 9 + df * thr))) - r
        total += stats.chi2.sf(max(0.0, root) ** 2, df)
    return total


@pytest.mark.parametrize("ntraits,nsnp", [(1, 3000), (1, 40000), (8, 250000), (8, 400000)])
@pytest.mark.parametrize("r", [0.3, 0.8, 1.0])
def test_the_candidates_that_are_expected_fit_their_lists(ctx, ntraits, nsnp, r):
    """The list of a segment stops at 2^22 entries however large the scan: with the share of candidates
    that the dispatch itself expects, no screened scan is thrown away and made again."""
    nid, t1, t2 = 8000, 5.7, 8.4
    ctx.lib.fake_traits(r, 0.002, 0.0)
    assert ctx.load(nid, nsnp) == capi.EPI_OK and ctx.traits(ntraits) == capi.EPI_OK
    ctx.lib.fake_rate(_share(t1, t2, "i", nid, nsnp * (nsnp - 1) / 2, r))
    st, n = ctx.scan(test="i", t1=t1, t2=t2, report_trait=-1, form=capi.FORM_TENSOR, tile_config=1)
    assert st == capi.EPI_OK and len({"full", "one", "two"} & set(n)) == 1
    assert n.get("one", 0) + n.get("two", 0) == n.get("exact", 0)


def test_what_a_scan_that_ran_over_says_of_others(ctx):
    """After a list ran over, a scan that asks for as much is made with all digits at once, without a
    second graph; one that asks for less (higher thresholds of the tests it makes, fewer pairs, one trait
    of many) is screened."""
    assert ctx.load(1000, 3000) == capi.EPI_OK and ctx.traits(2) == capi.EPI_OK
    f = dict(test="f", t1=8.0, t2=1.0, tile_config=1)
    ctx.lib.fake_traits(0.5, 0.002, 0.0)
    ctx.lib.fake_rate(0.05)
    assert ctx.scan(**f) == (capi.EPI_OK, {"one": 1, "exact": 1, "full": 1, "captures": 1})
    assert ctx.scan(**f) == (capi.EPI_OK, {"full": 1, "captures": 1})
    assert ctx.scan(**f) == (capi.EPI_OK, {"full": 1})
    ctx.lib.fake_rate(0.0)
    for same in (dict(t2=99.0), dict(t1=7.0), dict(report_trait=-1), dict(test="i", t2=99.0)):  # (8 df: t2 is not used)
        assert "one" not in ctx.scan(**dict(f, **same))[1], same
    for less in (dict(t1=8.5), dict(report_trait=1)):
        assert "full" not in ctx.scan(**dict(f, **less))[1], less
    assert "full" not in ctx.scan([(0, 300, 0, 300)], **f)[1]


@pytest.mark.parametrize("loads", [False, True], ids=["traits", "filesets"])
def test_a_loop_over_traits_that_run_over(ctx, loads):
    """Each step of a loop loads another trait (or fileset, too) for which the screen's list runs over: the
    screen is tried after 1, 2, 4 .. 64 steps, not in each; it is back within as many steps once the list
    holds, in every step from then on, and a cohort of another size starts afresh."""
    f = dict(t1=8.0, tile_config=1)
    assert ctx.load(1000, 3000) == capi.EPI_OK

    def steps(n):
        tried, captures = 0, 0
        for _ in range(n):
            assert not loads or ctx.load(1000, 3000) == capi.EPI_OK
            assert ctx.traits() == capi.EPI_OK
            for _ in range(2):  # (a second scan of the same data is never screened after the first ran over)
                st, k = ctx.scan(**f)
                assert st == capi.EPI_OK
                tried += k.get("one", 0)
                captures += k.get("captures", 0)
        return tried, captures
    ctx.lib.fake_rate(0.05)
    tried, captures = steps(200)
    assert 4 <= tried <= 10 and captures <= 2 * tried
    ctx.lib.fake_rate(0.0)
    steps(65)
    assert steps(10)[0] == 20
    ctx.lib.fake_rate(0.05)
    assert steps(2)[0] == 1
    assert ctx.load(900, 3000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    assert ctx.scan(**f)[1].get("one") == 1


def test_few_individuals_keep_the_plain_form_behind_the_screen(ctx):
    """The automatic form below 256 individuals is the plain one: where its pairs cannot be screened (low
    thresholds, a list that runs over, no memory, a tile shape of its own) and for the dump. From 64 on the
    tensor form screens it."""
    assert ctx.load(200, 5000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    ctx.lib.fake_traits(0.1, 0.001, 1.0)
    st, n = ctx.scan(**HIGH)
    assert st == capi.EPI_OK and n.pop("one") > 0 and set(n) == {"exact", "captures"}
    assert set(ctx.scan(**LOW)[1]) == {"plain", "captures"}
    assert set(ctx.scan(tile_config=2, **HIGH)[1]) == {"plain", "captures"}
    ctx.lib.fake_rate(0.05)
    assert set(ctx.scan(**HIGH)[1]) == {"one", "exact", "plain", "captures"}
    assert set(ctx.scan(**HIGH)[1]) == {"plain", "captures"}
    ctx.lib.fake_rate(0.0)
    assert "full" in ctx.scan(form=capi.FORM_TENSOR, **LOW)[1]
    assert ctx.load(63, 5000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    assert set(ctx.scan(**HIGH)[1]) == {"plain", "captures"}
    assert ctx.load(256, 5000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    assert "full" in ctx.scan(**LOW)[1]


def test_requested_variants_where_expanded_rows_do_not_fit(ctx):
    """Variant 3 streams B under the screen and does not without: where the rows do not fit it is refused no
    more than before there was a screen. Variant 6 streams B always, and is."""
    assert ctx.load(4000, 800000) == capi.EPI_OK and ctx.traits() == capi.EPI_OK
    ctx.lib.fake_limit(ctx.lib.fake_used() + (10 << 30))
    for k in range(1, 7):
        st, n = ctx.scan(form=capi.FORM_TENSOR, tile_config=k, **HIGH)
        if k == 6:
            assert (st, n) == (capi.EPI_E_UNSUPPORTED, {})
        else:
            assert st == capi.EPI_OK and ("full" if k == 3 else "one") in n and len({"full", "one"} & set(n)) == 1
