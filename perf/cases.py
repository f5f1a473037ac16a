"""The work that users have this library do, as cases that can be timed and compared.

A case scans SNP pairs through one of the public entry points (epigpu_b200.capi, the ctypes
binding of include/epigpu.h): `epi_scan` on a loaded context, `epi_set_phenotype` or the
whole upload before it, the plain form on request, and the allocation-free block scan.
Inputs are synthetic, from the package's own generator: Hardy-Weinberg genotypes with minor
allele frequencies of 0.05 to 0.5 and 1% of the calls missing, phenotypes N(0, 1) (right-
skewed gamma for every second trait of the multi-trait cases) with a few percent missing and
a few planted interactions, thresholds at p = 1e-6 as the benchmark's. Sizes are those of the
benchmark's configurations where they fit, else of the same kind, odd ones among them.

Keys of a case:
  kind    how the scan is called:
            scan      genotypes and traits loaded, epi_scan (a second threshold, another block
                      list: the call that every program makes)
            permute   the same with the columns of a permutation test: column 0 observed, the
                      others permuted copies under one missing mask, hits of column 0 only
            traits    several traits, each with its own missing mask, hits of every trait
            rephen    epi_set_phenotype, then epi_scan: one step of a loop over phenotypes
            load      epi_load_packed, epi_set_phenotype, epi_scan: a fileset just read
            plain     epi_scan with the plain form asked for (`-g p`)
            noalloc   epi_scan_block_noalloc on the caller's device buffers
  nid     individuals
  nsnp    SNPs in all
  nchr    chromosomes (every block of two of them is scanned, as the command line does),
          sizes falling by a constant factor to a twelfth of the largest where nchr > 2
  test    'f': 8 df; 'i': 8 df and 4 df
  ntraits phenotype columns
"""
import math

import numpy as np
import torch

from epigpu_b200 import capi, synth

P_VALUE = 1e-6  # of the two thresholds
CHUNK, SLOT = 128, 16  # iteration size of the output order and its slots a side (normal mode)


def listed():
    def c(name, kind, nid, nsnp, nchr=1, test="f", ntraits=1):
        return {"name": name, "kind": kind, "nid": nid, "nsnp": nsnp, "nchr": nchr, "test": test,
                "ntraits": ntraits}
    return [
        # a candidate-region look at a pilot cross: the smallest call, where latency counts
        c("pilot_n150", "scan", 150, 240),
        # an F2 cross of a model organism: a few hundred animals, a genome-wide marker panel
        c("cross_n231", "scan", 231, 2003, 3, "i"),
        # configuration 1 of the benchmark: the size that the reference's users run on a CPU
        c("small_n500", "scan", 500, 2000),
        # a cohort of about two thousand with a candidate panel, ragged everywhere
        c("cohort_n1999", "scan", 1999, 6001, 1, "i"),
        # configuration 2: two chromosomes, all three of their blocks
        c("twochr_n4000", "scan", 4000, 20000, 2, "i"),
        # configuration 3, the headline: one large chromosome, both tests
        c("large_n10000", "scan", 10000, 100000, 1, "i"),
        # configuration 4 with fewer SNPs: an observed trait and 63 permutations of it
        c("permute_n5000_t64", "permute", 5000, 4000, 1, "f", 64),
        # configuration 5 with fewer SNPs: 22 uneven chromosomes, 8 traits with own masks
        c("traits_n8000_t8", "traits", 8000, 10007, 22, "f", 8),
        # one step of a loop over phenotypes (an expression panel, the `-p` permutations)
        c("rephen_n3001", "rephen", 3001, 3000),
        # from a fileset just read to its hits: upload, unpacking and the traits included
        c("load_n2504", "load", 2504, 12000, 4, "i"),
        # the plain form, which `-g p` asks for, at configuration 2's individuals
        c("plain_n4000", "plain", 4000, 4001, 1, "i"),
        # a service that lends its own device buffers
        c("noalloc_n1203", "noalloc", 1203, 2502, 1, "i"),
    ]


def draw(rng):
    kind = rng.choice(["scan"] * 5 + ["permute", "traits", "rephen", "load", "plain", "noalloc"])

    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    nid = int(log(400 if kind in ("permute", "traits") else 100, 16000))
    # individuals x pairs x traits of the case; the CUDA-core forms do less in a given time
    top = {"scan": 4e13, "permute": 1e13, "traits": 1e13, "rephen": 1e12, "load": 4e12, "plain": 4e11,
           "noalloc": 4e10}[kind]
    work = log(min(1e8, top / 100), top)
    ntraits = {"permute": int(log(8, 128)), "traits": rng.randint(2, 12)}.get(kind, 1)
    nsnp = int(math.sqrt(2.0 * work / (nid * ntraits)))
    nsnp = max(100, min(100000 if nid >= 3000 else 30000, nsnp))
    if rng.random() < 0.3:
        nsnp = max(64, nsnp // 64 * 64)  # a round size now and then
    nchr = 1 if kind == "noalloc" or nsnp < 1000 else rng.choice([1, 1, 2, 5, 19, 22])
    return {"kind": kind, "nid": nid, "nsnp": nsnp, "nchr": nchr, "test": rng.choice("fi"), "ntraits": ntraits}


def chromosomes(case):
    n, m = case["nchr"], case["nsnp"]
    if n <= 2:
        sizes = [m // n] * n
    else:
        w = [12.0 ** (-c / (n - 1.0)) for c in range(n)]
        sizes = [max(1, int(m * x / sum(w))) for x in w]
    sizes[0] += m - sum(sizes)
    return sizes


def blocks_of(case):
    sizes = chromosomes(case)
    starts = np.cumsum([0] + sizes[:-1])
    return [(int(starts[i]), sizes[i], int(starts[j]), sizes[j]) for i in range(len(sizes)) for j in range(i + 1)]


def thresholds(case):
    nid = case["nid"]
    return synth.f_threshold(8, nid - 9, P_VALUE), synth.f_threshold(4, nid - 9, P_VALUE)


def capacity(case):
    """Rows of the program's hit buffer: several times what chance gives at these thresholds
    (more where skewed traits meet small cells). A scan with more hits fills it with the first."""
    return 512 + int(pairs_of(case) * case["ntraits"] * (1e-3 if case["kind"] == "traits" else 2e-5))


def inputs(case, seed):
    """Packed genotypes, phenotype columns (nid, T) and valid flags (None: -9 is missing)."""
    nid, nsnp, kind, ntraits = case["nid"], case["nsnp"], case["kind"], case["ntraits"]
    gpack = synth.packed_on_gpu(nid, nsnp, seed=1000 + seed)
    rng = np.random.default_rng(2000 + seed)
    if kind == "traits":
        cols, masks = [], []
        for t in range(ntraits):
            v = rng.standard_normal(nid) if t % 2 == 0 else (rng.gamma(2.0, 1.0, nid) - 2.0) / math.sqrt(2.0)
            cols.append(v.astype(np.float32))
            masks.append(rng.random(nid) >= rng.uniform(0.0, 0.10))
        return gpack, np.stack(cols, 1), np.stack(masks, 1)
    pairs = [tuple(int(x) for x in rng.choice(nsnp, 2, replace=False)) for _ in range(3)]
    rows = synth.planted_rows(gpack, nid, pairs)
    permuted = kind == "permute"
    y = synth.planted_phenotype(rows, pairs, seed=3000 + seed, var_frac=0.01, miss=0.0 if permuted else 0.01)
    if not permuted:
        return gpack, y[:, None], None
    cols = [y] + [capi.permute_phenotype(y, p) for p in range(1, ntraits)]
    valid = rng.random(nid) >= 0.01
    return gpack, np.stack(cols, 1), np.repeat(valid[:, None], ntraits, 1)


def prepare(case, seed):
    gpack, y, valid = inputs(case, seed)
    kind, nid, nsnp = case["kind"], case["nid"], case["nsnp"]
    t1, t2 = thresholds(case)
    opts = capi.default_opts(test=case["test"], t1=t1, t2=t2, chunk=CHUNK,
                             form=capi.FORM_POPC if kind == "plain" else capi.FORM_AUTO,
                             report_trait=-1 if kind == "traits" else 0)
    cap = capacity(case)
    state = {"case": dict(case), "opts": opts, "blocks": blocks_of(case), "cap": cap}
    if kind == "noalloc":
        state["gpack"] = torch.from_numpy(gpack).cuda()
        state["phen"] = torch.from_numpy(np.ascontiguousarray(y[:, 0])).cuda()
        state["hits"] = torch.zeros((cap, 6), dtype=torch.int32, device="cuda")
        state["nhits"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        state["maxf"] = torch.zeros(2, dtype=torch.float32, device="cuda")
        state["rows"] = torch.zeros((cap, 6), dtype=torch.int32, device="cuda")  # the same, sorted
        state["block"] = capi.Block(0, nsnp, 0, nsnp)
        return state
    ctx = capi.Context(0)
    ctx.load_packed(gpack, nid)
    ctx.set_traits(y, valid)
    state["ctx"] = ctx
    # the program's own table of hits, whose rows past the last hit stay zero
    state["pairs"] = np.zeros((cap, 6), dtype=np.int32)
    state["F"], state["F2"] = np.zeros(cap, dtype=np.float32), np.zeros(cap, dtype=np.float32)
    if kind == "load":
        state["gpack"] = gpack
    if kind in ("load", "rephen"):
        state["phen"] = np.ascontiguousarray(y[:, 0])
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        st = capi.load().epi_scan_block_noalloc(
            state["gpack"].data_ptr(), case["nid"], case["nsnp"], state["phen"].data_ptr(), state["block"],
            state["opts"], state["hits"].data_ptr(), state["hits"].shape[0], state["nhits"].data_ptr(),
            state["maxf"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != capi.EPI_OK:
            raise RuntimeError("epi_scan_block_noalloc: status %d" % st)
        n = int(state["nhits"])
        rows = state["hits"][:n]  # in no particular order: sorted by the caller
        state["rows"][:n] = rows[torch.argsort(rows[:, 0].long() * case["nsnp"] + rows[:, 1])]
        f = state["rows"][:, 4:].view(torch.float32)
        return {"pairs": state["rows"][:, :4], "F": f[:, 0], "F2": f[:, 1], "max": state["maxf"]}
    ctx = state["ctx"]
    if kind == "load":
        ctx.load_packed(state["gpack"], case["nid"])
    if kind in ("load", "rephen"):
        ctx.set_phenotype(state["phen"])
    hits, total, more = ctx.scan(state["blocks"], state["opts"], cap=state["cap"], ntraits=case["ntraits"],
                                 want_blocks=True, want_traits=True)
    n = len(hits)
    pairs = state["pairs"][:n]
    for k, field in enumerate(("snp1", "snp2", "df1", "df2")):
        pairs[:, k] = hits[field]
    pairs[:, 4], pairs[:, 5] = more["block"], more["trait"]
    state["F"][:n], state["F2"][:n] = hits["F"], hits["F2"]
    return {"pairs": state["pairs"], "F": state["F"], "F2": state["F2"], "total": total,
            "max_f": more["max_f"], "max_f2": more["max_f2"]}


def pairs_of(case):
    return case["nsnp"] * (case["nsnp"] - 1) // 2


def work(case):
    """Packed genotypes (2 bits a call) and phenotypes read once, hits written once; for every
    pair, individual and trait the nine cells' count and phenotype sum as a contraction (the
    counts as often as the masks differ)."""
    nid, nsnp, ntraits = case["nid"], case["nsnp"], case["ntraits"]
    masks = ntraits if case["kind"] == "traits" else 1
    steps = float(pairs_of(case)) * nid
    return {"bytes": nsnp * ((nid + 15) // 16 * 4.0) + 4.0 * nid * ntraits + 24.0,
            "flops": 2.0 * 9.0 * steps * (ntraits + masks)}


# ---- the same statistics in 64 bits ----

def _codes(gpack, nid):
    """(nsnp, nid) uint8 codes on the GPU from the packed rows."""
    w = torch.from_numpy(np.ascontiguousarray(gpack)).cuda()
    npack, remain = divmod(nid, 16)
    parts = []
    if npack:
        sh = torch.arange(30, -1, -2, device="cuda", dtype=torch.int32)
        parts.append(((w[:, :npack, None] >> sh) & 3).to(torch.uint8).reshape(w.shape[0], -1))
    if remain:
        sh = torch.arange(2 * (remain - 1), -1, -2, device="cuda", dtype=torch.int32)
        parts.append(((w[:, npack:npack + 1] >> sh) & 3).to(torch.uint8))
    return torch.cat(parts, 1)


def _tables(ci, cj, y, w):
    """Counts and sums of the 3 x 3 cells and the sum of squares of every pair of two groups of
    SNPs: (9, i, j) twice and (i, j), in 64 bits."""
    def rows(c, v):  # genotype-major indicator rows times v
        return torch.cat([(c == g).double() * v for g in range(3)])
    i, j = ci.shape[0], cj.shape[0]
    ones = torch.ones_like(y)
    a = rows(ci, ones)

    def cells(v):
        return (a @ rows(cj, v).T).reshape(3, i, 3, j).permute(0, 2, 1, 3).reshape(9, i, j)
    n, s = cells(w).round(), cells(y)
    q = (ci != 3).double() @ ((cj != 3).double() * (y * y)).T
    return n, s, q


def _stats(n, s, q, want_int):
    tot, st = n.sum(0), s.sum(0)
    nfac = (n > 0).sum(0)
    m = st / tot
    mc = torch.where(n > 0, s / n.clamp(min=1), torch.zeros_like(s))
    ssb = (n * (mc - m).square()).sum(0)
    d1, d2 = nfac - 1, tot - nfac
    msw = (q - st * m - ssb) / d2
    f = ssb / d1 / msw
    f2 = torch.zeros_like(f)
    if want_int:
        n3, s3 = n.reshape(3, 3, *f.shape), s.reshape(3, 3, *f.shape)
        row, col = s3.sum(1) / n3.sum(1).clamp(min=1), s3.sum(0) / n3.sum(0).clamp(min=1)
        t = mc.reshape(3, 3, *f.shape) - row[:, None] - col[None] + m
        f2 = (n3 * t.square()).sum((0, 1)) / 4.0 / msw
    return nfac, d1, d2, f, f2


def exact(case, seed):
    steps = float(pairs_of(case)) * case["ntraits"]
    if steps * case["nid"] > 4e12 or steps > 1.5e9:
        return None
    gpack, y, valid = inputs(case, seed)
    nid, ntraits, test = case["nid"], case["ntraits"], case["test"]
    t1, t2 = (float(np.float32(t)) for t in thresholds(case))
    codes = _codes(gpack, nid)
    blocks = blocks_of(case)
    report = range(ntraits) if case["kind"] == "traits" else [0]
    found = [np.zeros((0, 8))]
    top = np.full((2, ntraits), -np.inf)
    for t in range(ntraits):
        ok = valid[:, t] if valid is not None else y[:, t] != -9.0
        w = torch.from_numpy(ok.astype(np.float64)).cuda()
        yt = torch.from_numpy(np.where(ok, y[:, t], 0.0).astype(np.float64)).cuda()
        yt = torch.where(w > 0, yt - yt.sum() / w.sum(), torch.zeros_like(yt))
        for b, (s1, m1, s2, m2) in enumerate(blocks):
            step = max(1, min(m1, (1 << 24) // m2))
            for i0 in range(0, m1, step):
                i1 = min(m1, i0 + step)
                j1 = min(m2, s1 + i1 - 1 - s2)  # SNPs below every i of the group and no others
                if j1 <= 0:
                    continue
                n, s, q = _tables(codes[s1 + i0:s1 + i1], codes[s2:s2 + j1], yt, w)
                nfac, d1, d2, f, f2 = _stats(n, s, q, test == "i")
                gi = torch.arange(s1 + i0, s1 + i1, device="cuda")[:, None]
                gj = torch.arange(s2, s2 + j1, device="cuda")[None]
                none = torch.full_like(f, -np.inf)
                inside = gi > gj
                top[0, t] = max(top[0, t], float(torch.where(inside & ~f.isnan(), f, none).max()))
                top[1, t] = max(top[1, t], float(torch.where(inside & ~f2.isnan(), f2, none).max()))
                if t not in report:
                    continue
                hit = inside & (f > t1 if test == "f" else ((f > t1) | (f2 > t2)) & (nfac > 6))
                at = hit.nonzero()
                a, c = at[:, 0], at[:, 1]
                one = [torch.full_like(a, t), torch.full_like(a, b), a + i0, c, d1[a, c], d2[a, c], f[a, c], f2[a, c]]
                found.append(torch.stack([x.double() for x in one], 1).cpu().numpy())
    h = np.concatenate(found)
    block, gx, gy = (h[:, k].astype(np.int64) for k in (1, 2, 3))
    where = np.asarray(blocks, dtype=np.int64)
    snp1, snp2 = where[block, 0] + gx, where[block, 2] + gy
    if case["kind"] == "noalloc":
        order = np.lexsort((snp2, snp1))
    else:  # the output order: trait, block, result slot, chunk of either side, then the pair
        order = np.lexsort((gy, gx, gy // CHUNK, gx // CHUNK, gx % SLOT * SLOT + gy % SLOT, block, h[:, 0]))
    h, block, snp1, snp2 = h[order], block[order], snp1[order], snp2[order]
    noalloc, n = case["kind"] == "noalloc", capacity(case)
    pairs = np.zeros((n, 4 if noalloc else 6), dtype=np.int32)
    f, f2 = np.zeros(n), np.zeros(n)
    rows = [snp1, snp2, h[:, 4], h[:, 5]] + ([] if noalloc else [block, h[:, 0]])
    pairs[:len(h)] = np.stack(rows, 1)[:n]
    f[:len(h)], f2[:len(h)] = h[:n, 6], h[:n, 7]
    if test == "f":
        top[1] = 0.0
    if noalloc:
        return {"pairs": pairs, "F": f, "F2": f2, "max": top[:, 0]}
    return {"pairs": pairs, "F": f, "F2": f2, "total": len(h), "max_f": top[0], "max_f2": top[1]}
