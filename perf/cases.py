"""Performance cases: alignment work as a user's program runs it through
mpgpu.py (the ctypes binding of libmpgpu.so).

A pass of the iteration cases is one Gauss-Newton iteration of a job whose
records stay on the device: the data loop (local fits, accumulation of the
global matrix), the pre-sigmas of the steering's parameter lines added to the
diagonal, and the solution.  The other cases are a solution alone (a matrix
kept on the device), the first data loop of a new data set (structure passes,
upload, loop) and a batch of whole jobs through the resident server.

The data are the seeded generators' telescope, helix-barrel and broken-line
barrel tracks, with the modules, hits and resolutions of the named workloads of
mpgpu.gen_config; the seed of prepare() seeds the generator and the starting
parameters.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_KIND = {"telescope": 1, "barrel": 2, "brokenlines": 3}
_HUBER = 1.345
_FRESH_FACTOR = 16   # mpgpu_cfg flag: metsol 31 factorises its own matrix at every solve


def _mp():
    name = "millepede_ii_gb300_mpgpu"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(_ROOT, "millepede-ii_gb300", "mpgpu.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ------------------------------------------------------------------ cases
def _iteration(name, kind, nmod, ntracks, metsol, **kw):
    c = dict(name=name, work="iteration", kind=kind, nmod=nmod, ntracks=ntracks, metsol=metsol, sparse=metsol in (4, 5),
             constraints=True, presigma=True, errors=False, lhuber=0, outliers=0.0, mbandw=0)
    c.update(kw)
    return c


def listed():
    return [
        # the telescope workload (200 shifts, 2 constraints) by matrix inversion with parameter errors: the
        # smallest job, launches and synchronisations
        _iteration("telescope_200_inversion", "telescope", 20, 5_000, 1, errors=True, presigma=False),
        # a module-level alignment of a test-beam size by inversion, the method pede's users take up to a few
        # thousand parameters
        _iteration("telescope_1500_inversion", "telescope", 150, 20_000, 1, errors=True, presigma=False),
        # the same by decomposition (pede's own Cholesky form)
        _iteration("telescope_2000_cholesky", "telescope", 200, 30_000, 3, presigma=False),
        # FP64 blocked decomposition of a mid-size barrel (packed storage, 6 parameters per module)
        _iteration("barrel_6000_fp64", "barrel", 1_000, 50_000, 32),
        # the blocked inversion: parameter errors of a few thousand globals
        _iteration("barrel_4200_errors", "barrel", 700, 20_000, 12, constraints=False, errors=True),
        # the scaled telescope with the tensor-core decomposition, its own matrix factorised (first iteration
        # of a job): the largest dense solve of the benchmark
        _iteration("telescope_20000_mixed", "telescope", 2_000, 200_000, 31, presigma=False),
        # the flagship: 5,000 modules, 30,000 globals, sparse storage, MINRES; a first iteration
        _iteration("barrel_30000_400k", "barrel", 5_000, 400_000, 4),
        # a later iteration of it: down-weighting with outliers in the data, fewer records
        _iteration("barrel_30000_huber", "barrel", 5_000, 60_000, 4, lhuber=3, outliers=0.01),
        # uneven local fits (4 to 40 hits, up to 82 locals, bordered-band solution) into sparse storage
        _iteration("brokenlines_30000", "brokenlines", 5_000, 50_000, 4),
        # MINRES-QLP on a matrix kept on the device, odd size
        dict(_iteration("barrel_9000_qlp", "barrel", 1_501, 15_000, 5), work="solve"),
        # a new data set: device structure passes from page-locked records, upload, first loop
        dict(_iteration("barrel_new_data", "barrel", 5_000, 150_000, 0, sparse=True), work="newdata"),
        # six queued jobs of mixed sizes through the resident server, two iterations each
        dict(name="server_6_jobs", work="server", jobs=6, nmod=400, ntracks=20_000),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    what = rng.choice(["inversion", "cholesky", "fp64", "errors", "mixed", "minres", "huber", "brokenlines", "solve",
                       "newdata", "server"])
    tel = rng.random() < 0.5
    if what == "inversion":
        nmod = _log(rng, 20, 150)
        c = _iteration("", "telescope", nmod, max(2_500, nmod * _log(rng, 100, 250)), 1, errors=True, presigma=False)
    elif what == "cholesky":
        nmod = _log(rng, 20, 200)
        c = _iteration("", "telescope", nmod, max(2_500, nmod * _log(rng, 100, 250)), 3, presigma=False)
    elif what in ("fp64", "errors"):
        top = 6_000 if what == "fp64" else 4_200
        n = _log(rng, 600, top)
        metsol = 32 if what == "fp64" else 12
        # the generator needs at least 288 barrel modules (three per ring)
        if tel or n < 1_800:
            c = _iteration("", "telescope", n // 10, 20 * n // 10 * 10, metsol, constraints=what == "fp64",
                           errors=what == "errors")
        else:
            c = _iteration("", "barrel", n // 6, _log(rng, 10_000, 50_000), metsol, constraints=what == "fp64",
                           errors=what == "errors")
    elif what == "mixed":
        n = _log(rng, 1_000, 19_000)
        if tel or n < 1_800 or n > 9_000:
            c = _iteration("", "telescope", n // 10, 10 * n, 31, presigma=False)
        else:
            c = _iteration("", "barrel", n // 6, _log(rng, 10_000, 50_000), 31)
    elif what == "minres":
        c = _iteration("", "barrel", _log(rng, 300, 5_000), _log(rng, 10_000, 380_000), 4)
    elif what == "huber":
        c = _iteration("", rng.choice(["barrel", "telescope"]), _log(rng, 300, 2_000), _log(rng, 10_000, 100_000), 4,
                       lhuber=rng.choice([2, 3]), outliers=0.01)
    elif what == "brokenlines":
        c = _iteration("", "brokenlines", _log(rng, 400, 5_000), _log(rng, 5_000, 50_000), 4)
    elif what == "solve":
        c = dict(_iteration("", "barrel", _log(rng, 300, 2_500), _log(rng, 5_000, 30_000), rng.choice([4, 4, 5]),
                            mbandw=rng.choice([0, 0, 6])), work="solve")
    elif what == "newdata":
        c = dict(_iteration("", rng.choice(["barrel", "brokenlines"]), _log(rng, 300, 5_000), _log(rng, 5_000, 70_000),
                            0, sparse=True), work="newdata")
    else:
        c = dict(name="", work="server", jobs=rng.randint(2, 6), nmod=rng.randint(300, 400),
                 ntracks=_log(rng, 5_000, 20_000))
    del c["name"]
    return c


# ------------------------------------------------------------------ data
def _cfg(kind, nmod, ntracks, seed, outliers=0.0):
    common = dict(ntracks=ntracks, seed=seed, outlierFrac=outliers, threads=max(2, os.cpu_count() or 2))
    if kind == "telescope":
        return _mp().GenCfg(kind=1, nlayers=10, nmod=nmod, sigma1=0.005, sigma2=0.005, misal=0.01, **common)
    if kind == "barrel":
        return _mp().GenCfg(kind=2, nmod=nmod, sigma1=0.002, sigma2=0.008, misal=0.005, **common)
    return _mp().GenCfg(kind=3, nmod=nmod, minHits=4, maxHits=40, sigma1=0.002, sigma2=0.008, misal=0.005,
                        theta0=0.001, **common)


def _data(case, seed):
    return _mp().generate(_cfg(case["kind"], case["nmod"], case["ntracks"], 1_000 + seed, case["outliers"]))


def _mreqenf(case):
    return 5 if case["kind"] == "telescope" else 25


def _presigma(kind, labels):
    """Pre-sigma of each label: the scale of the generator's misalignments (the barrel's rotations are labels
    4 to 6 of each module)."""
    labels = np.asarray(labels)
    if kind == "telescope":
        return np.full(len(labels), 0.01)
    return np.where((labels - 1) % 6 < 3, 0.005, 5e-5)


def _start(case, seed, n):
    """Current parameters of the iteration: zero in the first one, of the order of the remaining
    misalignments in a later one."""
    if not case["lhuber"]:
        return np.zeros(n)
    return np.random.RandomState(seed % (1 << 31)).uniform(-2e-4, 2e-4, n) * (
        1.0 if case["kind"] == "telescope" else np.where(np.arange(n) % 6 < 3, 1.0, 1e-2))


class _State:
    """What the program keeps; closes its context or server when dropped."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for a in ("server", "ctx"):
            if getattr(self, a, None) is not None:
                getattr(self, a).close()
        for p in getattr(self, "pinned", ()):
            p.free()


def _server_jobs(case, seed):
    """(data, parameter lines) of each job: alternating barrel and broken-line detectors of growing sizes."""
    out = []
    for k in range(case["jobs"]):
        f = (k + 1) / case["jobs"]
        kind = "brokenlines" if k % 3 == 2 else "barrel"
        nmod = max(300, int(case["nmod"] * (0.75 + 0.25 * f)))
        nt = max(3_000, int(case["ntracks"] * f * (0.5 if kind == "brokenlines" else 1.0)))
        d = _mp().generate(_cfg(kind, nmod, nt, 1_000 + 17 * seed + k))
        labels = np.arange(1, len(d["truth"]) + 1, dtype=np.int32)
        out.append((kind, d, (labels, np.zeros(len(labels)), _presigma(kind, labels))))
    return out


def prepare(case, seed):
    mp = _mp()
    if case["work"] == "server":
        jobs = [mp.JobData(d, params=p, metsol=31, matsto=1, mitera=2, lhuber=3, mreqenf=25, mrestl=1e-13)
                for _, d, p in _server_jobs(case, seed)]
        return _State(case=case, server=mp.Server(max_active=4), jobs=jobs, ctx=None)
    d = _data(case, seed)
    ctx = mp.Context(flags=_FRESH_FACTOR)
    st = _State(case=case, ctx=ctx, data=d, mreqenf=_mreqenf(case))
    st.nlabels = len(d["truth"])
    if case["work"] == "newdata":
        st.pinned = [mp.PinnedArray(d[k]) for k in ("inder", "glder")]
        st.data = dict(d, inder=st.pinned[0].a, glder=st.pinned[1].a)
        return st
    S = mp.DeviceStructure(ctx, d, mreqenf=st.mreqenf, sparse=case["sparse"])
    ctx.set_layout(S, 2 if case["sparse"] else 1)
    st.cres = None
    if case["constraints"]:
        A = mp.constraint_matrix(d, S)
        ctx.set_constraints(A)
        st.cres = np.zeros(len(A))
    ctx.upload(S)
    st.data = None
    st.gpar = _start(case, seed, S.nTotal)
    st.opts = dict(nloopn=2 if case["lhuber"] else 1, lhuber=case["lhuber"])
    st.iv = np.arange(1, S.nVar + 1, dtype=np.int32)
    st.vlabels = S.labels[S.varIndex > 0]
    st.pre = _presigma(case["kind"], st.vlabels) ** -2.0
    ctx.set_preconditioner(case["mbandw"])
    if case["work"] == "solve":
        ctx.loopbf(st.gpar, **st.opts)
        ctx.mupdat(st.iv, st.iv, st.pre)
    return st


def _by_label(n, labels, a):
    """Values of some labels in the program's table of all n labels (1..n), as it keeps its constants."""
    out = np.zeros(n, a.dtype)
    out[labels - 1] = a
    return out


def _solve(st):
    c = st.case
    corr, err, _ = st.ctx.solve(c["metsol"], consResiduals=st.cres, rtol=1e-13, itnlim=2000, errors=c["errors"])
    out = dict(correction=_by_label(st.nlabels, st.vlabels, corr))
    if c["errors"]:
        out["errors"] = _by_label(st.nlabels, st.vlabels, err)
    return out


def run(state):
    st, c = state, state.case
    if c["work"] == "server":
        tickets = [st.server.submit(j) for j in st.jobs]
        for t in tickets:
            rc = st.server.wait(t)[0]
            if rc:
                raise RuntimeError("job failed (%d): %s" % (rc, st.server.last_error()))
        return [j.parameters()[1] for j in st.jobs]
    if c["work"] == "solve":
        return _solve(st)
    if c["work"] == "newdata":
        S = _mp().DeviceStructure(st.ctx, st.data, mreqenf=st.mreqenf)
        st.ctx.set_layout(S, 2)
        st.ctx.upload(S)
        r = st.ctx.loopbf(np.zeros(S.nTotal))
        n, v = st.nlabels, S.labels[S.varIndex > 0]
        # the structure in arrays of the size the program reserves for it
        offsets, columns = np.zeros(2 * (n + 1), np.int64), np.zeros(max(1 << 20, len(S.columns)), np.int32)
        offsets[:len(S.offsets)], columns[:len(S.columns)] = S.offsets, S.columns
        return dict(entries=_by_label(n, S.labels, S.counter), variable=_by_label(n, S.labels, S.varIndex),
                    offsets=offsets, columns=columns, vector=_by_label(n, v, r["gvec"]),
                    counts=_by_label(n, v, r["gcnt"]), chi2=r["chi2"], ndf=r["ndf"])
    r = st.ctx.loopbf(st.gpar, **st.opts)
    if c["presigma"]:
        st.ctx.mupdat(st.iv, st.iv, st.pre)
    return dict(_solve(st), vector=_by_label(st.nlabels, st.vlabels, r["gvec"]),
                counts=_by_label(st.nlabels, st.vlabels, r["gcnt"]), chi2=r["chi2"], ndf=r["ndf"])


# ------------------------------------------------------------------ work
def _loop_work(kind, ntracks):
    """Bytes of the record words and floating-point operations of the local fits and updates (mean record)."""
    if kind == "telescope":
        nw, nmeas, nloc, ng, nalg = 51, 10, 2, 1, 10
    elif kind == "barrel":
        nw, nmeas, nloc, ng, nalg = 313, 24, 5, 6, 72
    else:
        nw, nmeas, nloc, ng, nalg = 690, 84, 44, 6, 120
    f = 2.0 * (nmeas * (nloc + nloc * (nloc + 1) / 2) + nloc ** 3 + nmeas * ng * (ng + 1) / 2 + nmeas * ng * nloc +
               nalg * nloc ** 2 + nloc * nalg * (nalg + 1) / 2)
    if kind == "brokenlines":
        # the local matrix is a band: the factorisation and the products over the locals of each equation
        f = 2.0 * (nmeas * 21 + nloc * 36 + 36 * 22 * 8 + nalg * (nalg + 1) / 2 * 3)
    return 12.0 * nw * ntracks, f * ntracks


def work(case):
    if case["work"] == "server":
        b = f = 0.0
        for k in range(case["jobs"]):
            g = (k + 1) / case["jobs"]
            n = 6.0 * case["nmod"] * (0.75 + 0.25 * g)
            lb, lf = _loop_work("barrel", case["ntracks"] * g)
            b += 2 * (lb + 8 * n * n / 2)
            f += 2 * (lf + n ** 3 / 3)
        return {"bytes": b, "flops": f}
    n = float(case["nmod"]) * (10 if case["kind"] == "telescope" else 6)
    lb, lf = _loop_work(case["kind"], case["ntracks"])
    pairs = min(n / 6 * (n / 6 + 1) / 2, case["ntracks"] * 78.0, 35.0 * n / 6 * (1 + n / 3e4)) \
        if case["kind"] != "telescope" else min(n * (n + 1) / 2, n * 30)
    nmat = n * (n + 1) / 2 if not case["sparse"] else pairs * (36 if case["kind"] != "telescope" else 1)
    b, f = lb + 8 * nmat + 32 * n, lf
    if case["work"] == "solve":
        b, f = 8 * nmat, 0.0
    if case["metsol"] in (4, 5):
        f += 100 * 4 * nmat      # of the order of a hundred products
    elif case["metsol"] in (3, 31, 32):
        f += n ** 3 / 3
    elif case["metsol"] in (1, 12):
        f += n ** 3
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact values
class _Plain:
    """One job's records and its Gauss-Newton iteration in plain torch, FP64, on the GPU."""

    def __init__(self, kind, d, mreqenf):
        dev = "cuda"
        ptr = torch.from_numpy(d["recPtr"]).to(dev)
        ind = torch.from_numpy(d["inder"]).to(dev)
        val = torch.from_numpy(d["glder"]).to(dev)
        nrec, nw = len(ptr) - 1, len(ind)
        zero = ind == 0
        zero[ptr[:-1]] = False               # the first word of a record
        z = torch.nonzero(zero).flatten()
        head, sig = z[0::2].contiguous(), z[1::2].contiguous()   # value and sigma words of each measurement
        self.rec = torch.searchsorted(ptr, head, right=True) - 1
        self.value, self.sigma = val[head], val[sig]
        neq = len(head)
        eq = torch.cumsum(torch.zeros(nw, dtype=torch.int64, device=dev).index_fill_(0, head, 1), 0) - 1
        nsig = torch.cumsum(torch.zeros(nw, dtype=torch.int64, device=dev).index_fill_(0, sig, 1), 0)
        isL = (ind > 0) & (nsig == eq)
        isG = (ind > 0) & (nsig == eq + 1)
        self.lw = (eq[isL], ind[isL].long() - 1, val[isL])
        ge, gl, gv = eq[isG], ind[isG].long(), val[isG]
        labels, inv = torch.unique(gl, return_inverse=True)
        entries = torch.bincount(inv)
        var = entries >= mreqenf
        self.labels, self.variable = labels.cpu().numpy(), var.cpu().numpy()
        self.nvar = int(var.sum())
        index = torch.cumsum(var.long(), 0) - 1
        index[~var] = -1
        self.gw = (ge, inv, index[inv], gv)
        first = torch.searchsorted(self.rec, torch.arange(nrec, device=dev))
        self.eqIn = torch.arange(neq, device=dev) - first[self.rec]   # equation within the record
        self.nrec = nrec

    def loop(self, gpar, lhuber):
        """(matrix, vector, chi2) of one data loop with the parameters gpar (all labels, in order)."""
        dev, n = "cuda", self.nvar
        par = torch.as_tensor(gpar, device=dev)
        ge, gi, gvar, gv = self.gw
        le, li, lv = self.lw
        rm = self.value.clone().index_add_(0, ge, -gv * par[gi])
        A = torch.zeros(n * n, dtype=torch.float64, device=dev)
        vec = torch.zeros(n, dtype=torch.float64, device=dev)
        chi2 = 0.0
        nloc = torch.zeros(self.nrec, dtype=torch.int64, device=dev).scatter_reduce_(0, self.rec[le], li + 1, "amax")
        neq = torch.bincount(self.rec, minlength=self.nrec)
        order = torch.argsort(neq, stable=True)
        keep = gvar >= 0
        ge, gvar, gv = ge[keep], gvar[keep], gv[keep]
        pos = 0
        rank = torch.empty_like(order)
        rank[order] = torch.arange(self.nrec, device=dev)
        step0 = int(4e8 // max(1, int(neq.max()) * (int(neq.max()) * 4 + 1)))
        recL, recG, rkE = rank[self.rec[le]], rank[self.rec[ge]], rank[self.rec]
        soL, soG, soE = torch.argsort(recL, stable=True), torch.argsort(recG, stable=True), torch.argsort(rkE, stable=True)
        bL, bG, bE = recL[soL], recG[soG], rkE[soE]
        while pos < self.nrec:
            m = min(self.nrec - pos, max(256, step0))
            cut = torch.tensor([pos, pos + m], device=dev)
            cl, cg, ce = (torch.searchsorted(b, cut).tolist() for b in (bL, bG, bE))
            iL, iG, iE = soL[cl[0]:cl[1]], soG[cg[0]:cg[1]], soE[ce[0]:ce[1]]
            rows = order[pos:pos + m]
            ne, nl = int(neq[rows].max()), int(nloc[rows].max())
            r0, e0 = rkE[iE] - pos, self.eqIn[iE]
            r, s = (torch.zeros(m, ne, dtype=torch.float64, device=dev) for _ in range(2))
            r[r0, e0] = rm[iE]
            s[r0, e0] = self.sigma[iE]
            live = s > 0
            w0 = torch.where(live, 1.0 / torch.where(live, s, 1.0) ** 2, 0.0)
            L = torch.zeros(m, ne, nl, dtype=torch.float64, device=dev)
            L[recL[iL] - pos, self.eqIn[le[iL]], li[iL]] = lv[iL]
            pad = torch.diag_embed((torch.arange(nl, device=dev)[None] >= nloc[rows][:, None]).double())
            lc = torch.zeros_like(r)
            for it in range(1, (lhuber if lhuber else 1) + 1):
                w = w0
                if lhuber and it > 1:
                    a = (r - lc).abs()
                    w = torch.where(a > _HUBER * s, w0 * _HUBER * s / a.clamp_min(1e-300), w0)
                gam = torch.linalg.cholesky(L.mT @ (w[..., None] * L) + pad)
                lc = (L @ torch.cholesky_solve(L.mT @ (w * r)[..., None], gam))[..., 0]
            res = r - lc
            c2 = w0 * res * res
            if lhuber:
                p = res.abs() / torch.where(live, s, 1.0)
                c2 = torch.where((p > _HUBER) & live, 2 * _HUBER * (p - 0.5 * _HUBER), c2)
            chi2 += float(c2.sum())
            vec.index_add_(0, gvar[iG], gv[iG] * (w * res)[recG[iG] - pos, self.eqIn[ge[iG]]])
            # the record's variable parameters as columns
            key, slot = torch.unique((recG[iG] - pos) * n + gvar[iG], return_inverse=True)
            kr, kv = key // n, key % n
            f = torch.searchsorted(kr, torch.arange(m + 1, device=dev))
            ns = int((f[1:] - f[:-1]).max()) if len(key) else 0
            if ns:
                col = torch.arange(len(key), device=dev) - f[kr]
                G = torch.zeros(m, ne, ns, dtype=torch.float64, device=dev)
                G.index_put_((recG[iG] - pos, self.eqIn[ge[iG]], col[slot]), gv[iG], accumulate=True)
                ids = torch.full((m, ns), -1, dtype=torch.int64, device=dev)
                ids[kr, col] = kv
                wG = w[..., None] * G
                B = L.mT @ wG
                U = G.mT @ wG - B.mT @ torch.cholesky_solve(B, gam)
                ok = (ids[:, :, None] >= 0) & (ids[:, None, :] >= 0)
                A.index_add_(0, (ids[:, :, None] * n + ids[:, None, :])[ok], U[ok])
                del G, wG, B, U, ok
            pos += m
        return A.view(n, n), vec, chi2

    def solve(self, A, vec, pre, C):
        """Minimum of the quadratic form on the null space of the constraints, and the inverse's diagonal
        where there are none."""
        A = A.clone()
        if pre is not None:
            A.diagonal().add_(torch.as_tensor(pre, device=A.device))
        d = A.diagonal().clone().rsqrt()
        A *= d[:, None] * d[None, :]
        if C is not None:
            Cs = torch.as_tensor(C, device=A.device) * d
            Cs = torch.linalg.qr(Cs.mT)[0].mT.contiguous()
            A.addmm_(Cs.mT, Cs)     # A + C^T C: the same constrained minimum, and positive definite
        F = torch.linalg.cholesky(A)
        x = torch.cholesky_solve((d * vec)[:, None], F)
        if C is None:
            r = (d * vec)[:, None] - A @ x
            return (d * (x + torch.cholesky_solve(r, F))[:, 0]), torch.cholesky_inverse(F).diagonal() * d * d
        Y = torch.cholesky_solve(Cs.mT.contiguous(), F)

        def project(x):
            return x - Y @ torch.linalg.solve(Cs @ Y, Cs @ x)

        x = project(x)
        x = x + project(torch.cholesky_solve((d * vec)[:, None] - A @ x, F))
        return d * x[:, 0], None

    def constraints(self, d):
        """Constraint rows over the variable parameters."""
        pos = {int(lab): i for i, lab in enumerate(self.labels[self.variable])}
        C = np.zeros((d["ncon"], self.nvar))
        for k in range(d["ncon"]):
            for q in range(d["conStart"][k], d["conStart"][k + 1]):
                i = pos.get(int(d["conLabel"][q]))
                if i is not None:
                    C[k, i] += d["conCoef"][q]
        return C


def exact(case, seed):
    if case["work"] == "server":
        out = []
        for kind, d, par in _server_jobs(case, seed):
            P = _Plain(kind, d, 25)
            C = P.constraints(d)
            pre = _presigma(kind, P.labels[P.variable]) ** -2.0
            full = np.zeros(len(par[0]))
            at = P.labels - 1
            for it in range(2):
                A, vec, _ = P.loop(full[at], 3 if it else 0)
                full[at[P.variable]] += P.solve(A, vec, pre, C)[0].cpu().numpy()
            out.append(full)
        return out
    d = _data(case, seed)
    P = _Plain(case["kind"], d, _mreqenf(case))
    A, vec, chi2 = P.loop(_start(case, seed, len(P.labels)), case["lhuber"])
    n, v = len(d["truth"]), P.labels[P.variable]
    if case["work"] == "newdata":
        return dict(entries=None, variable=None, offsets=None, columns=None,
                    vector=_by_label(n, v, vec.cpu().numpy()), counts=None, chi2=chi2, ndf=None)
    pre = _presigma(case["kind"], v) ** -2.0 if case["presigma"] or case["work"] == "solve" else None
    C = P.constraints(d) if case["constraints"] else None
    x, inv = P.solve(A, vec, pre, C)
    out = dict(correction=_by_label(n, v, x.cpu().numpy()))
    if case["errors"]:
        # with constraints the reference's errors are not those of the constrained covariance
        out["errors"] = _by_label(n, v, inv.cpu().numpy()) if C is None else None
    if case["work"] == "iteration":
        out.update(vector=_by_label(n, v, vec.cpu().numpy()), counts=None, chi2=chi2, ndf=None)
    return out
