"""The work a user of this library has it do, as cases that can be timed.

The sizes are the repository's own configurations (``eimp_b200/synth.py``): a
5,000-haplotype panel for the plain form, 10,000 haplotypes for the full
phase + impute run, 20,000 for batches of several array densities and for
serving, 200,000 for the large panel; K, beam width, typed densities and
missingness as there.  Panels and targets are Li-Stephens mosaics drawn on the
device from the seed alone (``eimp_b200/synth_device.py``).

Kinds:

* ``phase``   Target::prepPhase + Target::phase of a batch: best haplotypes,
  condensed reference, PBWTs, beam.  ``host`` takes numpy arrays through
  ``Phaser.phase``; otherwise the batched form on device buffers
  (``DensityGroup.phase``).
* ``impute``  match search and dosages of a batch against a resident
  reference (``DensityGroup.impute``).
* ``build``   the same after building the imputation reference of a new
  typed-site set (``DensityGroup.set_reference``), as every new array or
  window needs.
* ``output``  ``impute`` and the numbers the writer puts into its records
  (``eimp_imp_site_stats_dev``).
* ``serve``   one serving request from host genotypes to host dosages
  (``WindowSlot.run``).
* ``qref``    the haplotype section of a Qref panel file decoded from host
  memory into the resident panel (``eimp_qref_decode``).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from eimp_b200 import synth_device
from eimp_b200._lib import EimpSiteStatsOpts, ptr
from eimp_b200.batch import DensityGroup
from eimp_b200.bits import W, transpose_bits
from eimp_b200.engine import Context, PhaseParams, Phaser
from eimp_b200.serving import WindowSlot
from eimp_b200.synth import SynthConfig, WindowRequest

DEV = "cuda"


def _phase(name, haps, sites, mb, founders, targets, K, beam, host, hsize=100, prephase=False, reverse=True,
           miss=0.02):
    c = dict(kind="phase", haps=haps, sites=sites, mb=mb, founders=founders, targets=targets, K=K, beam=beam,
             host=host, hsize=hsize, prephase=prephase, reverse=reverse, miss=miss)
    return dict(name=name, **c) if name else c


def _impute(name, kind, haps, sites, mb, founders, targets, typed, errors=0, calls=False, miss=0.02):
    c = dict(kind=kind, haps=haps, sites=sites, mb=mb, founders=founders, targets=targets, typed=typed,
             errors=errors, calls=calls, miss=miss)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # one new sample against the plain configuration's panel: latency
        _phase("phase_single", 5000, 2000, 5.0, 200, 1, 1024, 64, True, miss=0.01),
        # the plain configuration: 100 samples, host buffers in and out
        _phase("phase_cohort", 5000, 2000, 5.0, 200, 100, 1024, 64, True, miss=0.01),
        # the fast pre-phasing pass, forward only, a short history, odd sizes
        _phase("phase_options", 2998, 1203, 3.0, 120, 37, 777, 50, True, hsize=77, prephase=True, reverse=False,
               miss=0.03),
        # the full phase + impute configuration's batch: every warp slot taken
        _phase("phase_array", 10000, 5000, 20.0, 500, 1000, 4096, 128, False),
        # a share of the densest array's targets over a 40 Mb segment: long walks, few targets
        _phase("phase_dense", 20000, 32000, 40.0, 1000, 192, 4096, 128, False),
        # the large panel: the search for the best haplotypes weighs most here
        _phase("phase_large_panel", 200000, 10000, 30.0, 2500, 96, 8192, 128, False, miss=0.01),
        # match search and dosages of an array's batch, reference resident
        _impute("impute_array", "impute", 10000, 100000, 20.0, 500, 500, 0.05),
        # a bunch imputed and its records' numbers (ADS, GT, DS, GP, AF, MAF, r2, AC, AN)
        _impute("impute_output", "output", 5000, 20000, 5.0, 200, 200, 0.10, miss=0.01),
        # a new typed-site set of the 20,000-haplotype panel and a small batch on it
        _impute("impute_new_sites", "build", 20000, 100000, 10.0, 1000, 64, 0.03),
        # the same for the large panel
        _impute("impute_large_panel", "build", 200000, 100000, 6.0, 1000, 32, 0.02, miss=0.01),
        # one serving request: a 4 Mb window, typed, phased and imputed, host to host
        dict(name="serve_request", kind="serve", haps=20000, sites=40000, mb=4.0, founders=1000, targets=75,
             typed=0.03, K=4096, beam=128, miss=0.02),
        # loading a panel
        dict(name="qref_load", kind="qref", haps=10000, sites=20000, mb=4.0, founders=500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("phase", "phase", "phase", "impute", "output", "build", "serve", "qref"))
    haps = 2 * _log(rng, 300, 20000)
    founders = max(20, haps // 20)
    miss = round(rng.uniform(0.0, 0.05), 4)
    if kind == "phase":
        sites = _log(rng, 300, 12000)
        host = rng.random() < 0.5
        # the walk is sequential in the sites, the batch is limited by the condensed references
        targets = _log(rng, 1, max(2, min(1000, 4000000 // sites)))
        return _phase(None, haps, sites, round(sites * rng.uniform(0.0008, 0.004), 3), founders, targets,
                      _log(rng, 64, 8192), rng.choice((32, 50, 64, 100, 128)), host,
                      hsize=rng.choice((50, 77, 100, 100, 128)), prephase=host and rng.random() < 0.3,
                      reverse=rng.random() < 0.8, miss=miss)
    sites = _log(rng, 2000, 100000)
    mb = round(sites * rng.uniform(0.0001, 0.0002), 3)
    if kind == "qref":
        return dict(kind="qref", haps=min(haps, 30000), sites=min(sites, 20000), mb=mb, founders=founders)
    typed = round(rng.uniform(0.01, 0.08), 4)
    if kind == "serve":
        sites = min(sites, 60000)
        return dict(kind="serve", haps=haps, sites=sites, mb=mb, founders=founders, targets=_log(rng, 1, 150),
                    typed=typed, K=_log(rng, 256, 4096), beam=rng.choice((64, 128)), miss=miss)
    targets = _log(rng, 1, max(2, min(500, 20000000 // sites)))
    return _impute(None, kind, haps, sites, mb, founders, targets, typed,
                   errors=rng.choice((0, 0, 0, 1)) if targets <= 100 and typed * sites <= 2000 else 0,
                   calls=rng.random() < 0.25, miss=miss)


# ------------------------------------------------------------------ inputs
def _panel(case, seed):
    cfg = SynthConfig("drawn", nhaps=case["haps"], nsites=case["sites"], segment_mb=case["mb"],
                      founders=case["founders"], maf_min=max(5e-6, 0.5 / case["haps"]), seed=1000 + 7919 * seed)
    ctx = Context(0)
    panel = synth_device.generate(cfg, 0, ctx)
    ctx.close()
    return panel


def _targets(panel, typed, n, miss, seed):
    """n held-out targets at the typed sites: genotypes (n, M) uint8 with 3 =
    missing, and their true haplotypes (2n, M) uint8."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(31 + 104729 * seed)
    d_typed = torch.from_numpy(typed).to(DEV)
    th = torch.empty((2 * n, len(typed)), dtype=torch.uint8, device=DEV)
    for a in range(0, 2 * n, 1024):
        b = min(2 * n, a + 1024)
        words = synth_device.mosaics(gen, panel.d_founders, panel.d_cm, b - a, panel.cfg.mean_segment_cm,
                                     panel.cfg.copy_err)
        th[a:b] = ((words[:, d_typed >> 6] >> (d_typed & 63)) & 1).to(torch.uint8)
    gt = th[0::2] + th[1::2]
    gt[torch.rand(gt.shape, generator=gen, device=DEV) < miss] = 3
    # genotyping errors as arrays make them
    err = (torch.rand(gt.shape, generator=gen, device=DEV) < 0.0005) & (gt != 3)
    gt = torch.where(err, (gt + 1) % 3, gt)
    return gt.contiguous(), th, gen


def _phased(gt, th, gen):
    """Phased haplotypes as phasing leaves them: the targets' own with a few
    switches per chromosome segment, consistent with the genotypes; missing
    sites reference alleles.  (2n, W(M)) int64 words on the device."""
    n, M = gt.shape
    sw = torch.rand((n, M), generator=gen, device=DEV) < 8.0 / max(M, 8)
    par = (torch.cumsum(sw.to(torch.int32), 1) & 1).bool()
    m0 = torch.where(par, th[1::2], th[0::2])
    het, hom = gt == 1, gt == 2
    mat = torch.where(het, m0, hom.to(torch.uint8))
    pat = torch.where(het, 1 - m0, hom.to(torch.uint8))
    out = torch.stack((mat, pat), 1).reshape(2 * n, M)
    words = torch.zeros((2 * n, W(M)), dtype=torch.int64, device=DEV)
    for a in range(0, 2 * n, 256):
        words[a:a + 256] = synth_device.pack_bits(out[a:a + 256] != 0, W(M))
    return words


def _typed_sites(case, seed):
    rng = np.random.default_rng(77 + 15485863 * seed)
    m = max(2, int(round(case["typed"] * case["sites"])))
    return np.sort(rng.choice(case["sites"], m, replace=False)).astype(np.int64)


def _params(case):
    return PhaseParams(K=case["K"], beamwidth=case["beam"], hsize=case.get("hsize", 100),
                       doPrePhasing=case.get("prephase", False), doRevPhasing=case.get("reverse", True))


def _group(case, panel, typed, gt, params):
    g = DensityGroup(0, panel.d_site, panel.d_af, panel.nhaps, typed, None, None,
                     panel.cm[typed].astype(np.float32), gt.cpu().numpy(), params, batch_targets=gt.shape[0])
    return g


class _State:
    """What a program keeps between calls; closes its library context."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        torch.cuda.synchronize()
        self.owner.close()


def _imputation_inputs(case, seed):
    panel = _panel(case, seed)
    typed = _typed_sites(case, seed)
    gt, th, gen = _targets(panel, typed, case["targets"], case["miss"], seed)
    return panel, typed, gt, _phased(gt, th, gen), gen


def prepare(case, seed):
    kind = case["kind"]
    if kind == "qref":
        panel = _panel(case, seed)
        ctx = Context(0)
        sec = _qref_section(panel.d_site)
        out = torch.zeros_like(panel.d_site)
        torch.cuda.synchronize()
        return _State(owner=ctx, kind=kind, sec=sec, out=out, sites=case["sites"], samples=case["haps"] // 2)
    if kind == "phase":
        panel = _panel(case, seed)
        typed = np.arange(case["sites"], dtype=np.int64)
        gt, _, _ = _targets(panel, typed, case["targets"], case["miss"], seed)
        params = _params(case)
        if case["host"]:
            ctx = Context(0)
            site = panel.d_site.cpu().numpy().view(np.uint64)
            ph = Phaser(ctx, transpose_bits(site, panel.nsites, panel.nhaps), site, panel.cm.astype(np.float32))
            torch.cuda.synchronize()
            return _State(owner=ctx, kind=kind, host=True, ph=ph, params=params, gt=gt.cpu().numpy())
        g = _group(case, panel, typed, gt, params)
        torch.cuda.synchronize()
        return _State(owner=g, kind=kind, host=False)
    if kind == "serve":
        panel = _panel(case, seed)
        typed = _typed_sites(case, seed)
        gt, _, _ = _targets(panel, typed, case["targets"], case["miss"], seed)
        slot = WindowSlot(0, panel.d_site, panel.d_af, panel.cm, panel.nhaps, _params(case))
        torch.cuda.synchronize()
        return _State(owner=slot, kind=kind, req=WindowRequest(0, case["sites"], typed, gt.cpu().numpy()))
    panel, typed, gt, phased, gen = _imputation_inputs(case, seed)
    # the phasing parameters size the group's phasing buffers only
    g = _group(case, panel, typed, gt, PhaseParams(K=64, beamwidth=16))
    g.d_ph.copy_(phased.view(g.d_ph.shape))
    s = _State(owner=g, kind=kind, errors=case["errors"], calls=int(case["calls"]))
    if kind == "output":
        nt, ns = g.nt, g.Mref
        s.pdos = _phased_dosages(gt, phased, gen)
        f = dict(dtype=torch.float32, device=DEV)
        s.ads = torch.empty((2 * nt, ns), **f)
        s.gtbits = torch.zeros((2 * nt, g.ldb), dtype=torch.int64, device=DEV)
        s.ds = torch.empty((nt, ns), **f)
        s.gp = torch.empty((3 * nt, ns), **f)
        s.site = [torch.empty(ns, **f) for _ in range(3)]
        s.cnt = [torch.empty(ns, dtype=torch.int32, device=DEV) for _ in range(2)]
        s.ok = torch.empty(ns, dtype=torch.uint8, device=DEV)
        s.conflicts = torch.zeros(1, dtype=torch.int64, device=DEV)
        s.opts = EimpSiteStatsOpts(0, 0, 0.3, 0.0)
    torch.cuda.synchronize()
    if kind != "build":
        g.set_reference()
        g.ctx.synchronize()
    return s


def _phased_dosages(gt, phased, gen):
    """Mat and pat dosages as phasing returns them: 0 or 1 at homozygous
    sites, the phase confidence at heterozygous ones, 0 where missing."""
    n, M = gt.shape
    sh = torch.arange(M, device=DEV)
    mat = ((phased[0::2][:, sh >> 6] >> (sh & 63)) & 1).to(torch.float32)
    conf = 0.5 + 0.5 * torch.rand((n, M), generator=gen, device=DEV)
    het = gt == 1
    dm = torch.where(het, torch.where(mat > 0, conf, 1 - conf), (gt == 2).to(torch.float32))
    dp = torch.where(het, torch.where(mat > 0, 1 - conf, conf), (gt == 2).to(torch.float32))
    return dm.contiguous(), dp.contiguous()


def _qref_section(d_site):
    """The haplotype section of a Qref file for the rows: per variant its
    code's length (u64, 0: the raw row follows) and its run lengths,
    alternating from zeros, one byte below 128, else the low 7 bits with the
    high bit set and the next 8 bits."""
    rows, nw = d_site.shape
    nb = nw * 64
    shift = torch.arange(64, device=DEV)
    parts = []
    for r0 in range(0, rows, 2048):
        bits = ((d_site[r0:r0 + 2048, :, None] >> shift) & 1).to(torch.bool).reshape(-1, nb)
        n = bits.shape[0]
        change = torch.empty((n, nb + 1), dtype=torch.bool, device=DEV)
        change[:, 0] = bits[:, 0]                     # a first run of no zeros
        change[:, 1:nb] = bits[:, 1:] != bits[:, :-1]
        change[:, nb] = True                          # the end of the last run
        r, e = torch.nonzero(change, as_tuple=True)
        first = torch.ones_like(r, dtype=torch.bool)
        first[1:] = r[1:] != r[:-1]
        prev = torch.where(first, torch.zeros_like(e), torch.roll(e, 1))
        length = (e - prev).cpu().numpy()
        size = np.where(length < 128, 1, 2)
        r = r.cpu().numpy()
        code = np.zeros(int(size.sum()), np.uint8)
        at = np.concatenate(([0], np.cumsum(size)[:-1]))
        code[at] = np.where(length < 128, length, (length & 0x7F) | 0x80)
        two = size == 2
        code[at[two] + 1] = length[two] >> 7
        total = np.bincount(r, weights=size, minlength=n).astype(np.int64)
        begin = np.concatenate(([0], np.cumsum(total)))
        raw = d_site[r0:r0 + 2048].cpu().numpy().view(np.uint8)
        for i in range(n):
            if total[i] >= nb // 8:
                parts += [np.zeros(8, np.uint8), raw[i]]
            else:
                parts += [np.array([total[i]], np.uint64).view(np.uint8), code[begin[i]:begin[i + 1]]]
    return np.concatenate(parts)


# ------------------------------------------------------------------ one pass
def run(state):
    s = state
    if s.kind == "qref":
        ctx = s.owner
        ctx.check(ctx.L.eimp_qref_decode(ctx.h, ptr(s.sec), s.sec.size, s.sites, s.samples, s.out.data_ptr(),
                                         s.out.shape[1], None))
        return s.out
    if s.kind == "phase" and s.host:
        return s.ph.phase(s.params, s.gt)
    if s.kind == "serve":
        return s.owner.run(s.req)
    g = s.owner
    if s.kind == "phase":
        g.phase()
        return g.d_mats, g.d_pats, g.d_pdm, g.d_pdp, g.d_tc, g.d_nc
    if s.kind == "build":
        g.set_reference()
    g.impute(s.errors, s.calls)
    if s.kind != "output":
        return {"bits": g.d_bits, "dos": g.d_dos}
    ns = g.Mref
    r2, af, maf = s.site
    g.ctx.check(g.L.eimp_imp_site_stats_dev(
        g.h, 0, ns, g.d_bits.data_ptr(), g.ldb, g.d_dos.data_ptr(), ns, s.pdos[0].data_ptr(), s.pdos[1].data_ptr(),
        g.M, C.byref(s.opts), s.ads.data_ptr(), ns, s.gtbits.data_ptr(), g.ldb, s.ds.data_ptr(), s.gp.data_ptr(),
        r2.data_ptr(), af.data_ptr(), maf.data_ptr(), s.cnt[0].data_ptr(), s.cnt[1].data_ptr(), s.ok.data_ptr(),
        s.conflicts.data_ptr()))
    return {"bits": g.d_bits, "dos": g.d_dos, "ads": s.ads, "gtbits": s.gtbits, "ds": s.ds, "gp": s.gp, "r2": r2,
            "af": af, "maf": maf, "ac": s.cnt[0], "an": s.cnt[1], "pass": s.ok}


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    the genotype-haplotype comparisons that choose the conditioning
    haplotypes (one multiply-add each as a contraction)."""
    kind, nh, n = case["kind"], case["haps"], case["targets"] if "targets" in case else 0
    if kind == "qref":
        return {"bytes": 1.3 * case["sites"] * W(nh) * 8, "flops": 0}
    M = case["sites"] if kind == "phase" else max(2, int(round(case["typed"] * case["sites"])))
    phase = nh * M / 8 + n * M + n * (2 * W(M) * 8 + 8 * M + 8)
    if kind == "phase":
        return {"bytes": phase, "flops": 2.0 * n * nh * M}
    S = case["sites"]
    out = 2 * n * (4 * S + S / 8)
    panel = nh * S / 8
    impute = panel + 4 * S + n * M + 2 * n * W(M) * 8 + out
    if kind == "serve":
        return {"bytes": phase + impute, "flops": 2.0 * n * nh * M}
    if kind == "output":
        impute += 2 * n * (4 * S + S / 8) + n * 16 * S + 2 * n * 4 * M + 21 * S
    return {"bytes": impute, "flops": 0}


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    """Imputation by definition, in 64 bits.  Phasing has no such value: which
    paths its beam keeps depends on 32-bit sums."""
    if case["kind"] not in ("impute", "build", "output") or case["errors"]:
        return None
    n, M = case["targets"], max(2, int(round(case["typed"] * case["sites"])))
    if 2.0 * n * case["haps"] * M > 6e9 or 2.0 * n * M > 1.0e6 or 2.0 * n * case["sites"] > 2e7:
        return None
    panel, typed, gt, phased, gen = _imputation_inputs(case, seed)
    N, S = panel.nhaps, panel.nsites
    site = panel.d_site
    words = torch.empty((S, site.shape[1]), dtype=torch.int64).copy_(site).numpy().view(np.uint8)
    hap = torch.arange(N, device=DEV)
    rows = site[torch.from_numpy(typed).to(DEV)]
    refs = ((rows[:, hap >> 6] >> (hap & 63)) & 1).to(torch.bool).T.contiguous()      # (N, M)
    af = panel.d_af.cpu().numpy()
    minor = np.where(af > np.float32(0.5), np.float32(1) - af, af).astype(np.float32)
    rare = (minor * np.float32(N)).astype(np.float32).astype(np.float64)
    major = af > 0.5
    seg = np.maximum(np.searchsorted(typed, np.arange(S), side="right") - 1, 0)
    idx = torch.arange(M, device=DEV, dtype=torch.int32)
    pos = torch.arange(M, device=DEV)
    gth = gt.cpu().numpy()
    dos = np.empty((2 * n, S))
    for h in range(2 * n):
        own = ((phased[h, pos >> 6] >> (pos & 63)) & 1).to(torch.bool)
        missing = gt[h // 2] == 3
        # per haplotype of the panel, the last mismatch at or before every site
        last = torch.cummax(torch.where((refs != own) & ~missing, idx, -1), 1).values
        best = last.min(0).values.cpu().numpy() + 1         # start of the longest match through site m
        score, total = np.zeros(S), np.zeros(S)
        if int(missing.sum()) <= M // 2:
            end = [m for m in range(M) if (best[m + 1] > best[m] if m + 1 < M else True) and best[m] <= m]
            for m in end:
                a, e = int(best[m]), m + 1
                who = torch.nonzero(last[:, m] + 1 == a).flatten()
                mi = np.flatnonzero(gth[h // 2, a:e] == 3) + a
                # panel haplotypes that differ where the target is missing are separate matches
                height = np.full(len(who), len(who))
                if len(mi) and len(who) > 1:
                    pat = refs[who][:, torch.from_numpy(mi).to(DEV)].cpu().numpy()
                    _, inv, num = np.unique(pat, axis=0, return_inverse=True, return_counts=True)
                    height = num[inv.reshape(-1)]
                who = who.cpu().numpy()
                s0 = int(typed[a]) if a else 0
                s1 = int(typed[e]) if e < M else S
                k = seg[s0:s1]
                single = (k - a + 1.0) * (e - k)
                alt = (words[s0:s1][:, who >> 3] >> (who & 7)) & 1
                short = rare[s0:s1, None] < 0.01 * height[None, :]
                score[s0:s1] += single * np.where(short, major[s0:s1, None], alt).sum(1)
                total[s0:s1] += single * len(who)
        d = np.where(total > 0, score / np.maximum(total, 1), -1.0)
        if not case["calls"]:
            keep = typed[gth[h // 2] != 3]
            o = own.cpu().numpy()[gth[h // 2] != 3]
            d[keep] = o
        dos[h] = d
    if case["kind"] != "output":
        return {"bits": None, "dos": dos}
    dm, dp = (x.cpu().numpy().astype(np.float64) for x in _phased_dosages(gt, phased, gen))
    ads = np.where(dos < 0, af.astype(np.float64)[None, :], dos)
    for t in range(n):
        call = gth[t] != 3
        ads[2 * t, typed[call]] = dm[t, call]
        ads[2 * t + 1, typed[call]] = dp[t, call]
    a0, a1 = ads[0::2], ads[1::2]
    gp = np.stack(((1 - a0) * (1 - a1), a0 + a1 - 2 * a0 * a1, a0 * a1), 1).reshape(3 * n, S)
    mean = ads.mean(0)
    evar = mean * (1 - mean)
    ovar = (ads ** 2).mean(0) - mean ** 2
    r2 = np.where((evar > 1e-12) & (ovar > 1e-12), ovar / np.maximum(evar, 1e-300), 0.0)
    return {"bits": None, "dos": dos, "ads": ads, "gtbits": None, "ds": a0 + a1, "gp": gp, "r2": r2, "af": mean,
            "maf": np.minimum(mean, 1 - mean), "ac": None, "an": None, "pass": None}
