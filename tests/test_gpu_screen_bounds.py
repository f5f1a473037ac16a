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
