"""Timed cases of the fast search path, through the package's public entry
points.

Each case is one call (or the short chain of calls) that a search program
makes per page, cube or block:

  corr      FastCorrKernel.compute_raw on on-wire pages
  calcorr   unpack_int4_split -> apply_cal_split -> FastCorrKernel.compute_split
  stage1    Stage1MultiDMCoarseDM.dedisperse_from_vis (sliding window)
  imager    GpuImager.process_cube, dense or compact streams
  image     SearchPipeline.image from a filled stage-2 ring
  search    Layer-1, detect_images, Layer-2 and the candidate read-back
  boxcar    precompute_padded_cumsum -> multi_boxcar_argmax_triton
  pipeline  SearchPipeline.process_block, a whole streaming block

Sizes are those of the repository's benchmark workloads, tests and the
instrument's native pages (2048 packets, 96 antennas, 384 channels).
"""

import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "dsa110-rt_b200"))

from dsb200 import corr, dedisp, grid, pipeline, search, synth  # noqa: E402
from dsb200.constants import DSA110_BAND, Band, band_from_edges  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # the smallest correlator call: a 16-antenna test array's short page
        dict(name="corr-small", kind="corr", n_g=1, npkt=64, nant=16, nchan=128, t_int=8, csf=4,
             layout="tbc"),
        # one native page at the search cadence
        dict(name="corr-page", kind="corr", n_g=1, npkt=2048, nant=96, nchan=384, t_int=32,
             csf=16, layout="tbc"),
        # the calibrated chain on one native page
        dict(name="calcorr-page", kind="calcorr", npkt=2048, nant=96, nchan=384, t_int=32, csf=16,
             dtype="f16", fuse=True),
        # stage 1 of one chgroup's page at the 262-us cadence, 32 coarse DMs
        dict(name="stage1-page", kind="stage1", nant=96, n_fv=512, chgroup=15, csf=16, t_int=8,
             n_coarse=32, dm_max=2000.0, n_grid=256),
        # the imager on dense and on compact cint8 streams, half cubes
        dict(name="imager-dense-256", kind="imager", compact=False, n_grid=256, n_g=16, t_det=64,
             n_fdm=8, cube="f16", fill=4000),
        dict(name="imager-compact-256", kind="imager", compact=True, n_grid=256, n_g=16, t_det=64,
             n_fdm=16, cube="f16", fill=4000),
        # the streaming imager at the metric configuration's grid (one coarse
        # DM's 16 fine DMs, a quarter of a cube's times) and at 256^2
        dict(name="image-512-bf16", kind="image", n_grid=512, nant=96, n_chgroup=16, t_int=32,
             ring="bf16", dm_max=50.0, n_f=16, n_t=144),
        dict(name="image-256-c64", kind="image", n_grid=256, nant=96, n_chgroup=16, t_int=8,
             ring="c64", dm_max=50.0, n_f=8, n_t=272),
        # the search of a cube, boxcars 1..64 on 512^2
        dict(name="search-512-b64", kind="search", n_grid=512, n_f=8, n_out=256, logw=6),
        # the reference's two-step boxcar form on a half cube
        dict(name="boxcar-256-b16", kind="boxcar", n_grid=256, n_f=4, n_t=144, n_out=128, logw=4,
             cube="f16"),
        # a whole block of the small plain configuration (16 antennas, 64^2,
        # 32 DMs 0-600): latency and launches
        dict(name="block-64", kind="pipeline", n_grid=64, nant=16, n_chgroup=2, nchan=128, csf=4,
             t_int=8, npkt=2048, chunk=512, n_coarse=32, fine=1, dm_max=600.0, logw=4,
             ring="c64", batch=32),
        # a quarter block of the metric configuration over 128 of its DMs
        dict(name="block-512", kind="pipeline", n_grid=512, nant=96, n_chgroup=16, nchan=384,
             csf=16, t_int=32, npkt=2048, chunk=128, n_coarse=8, fine=16, dm_max=190.0, logw=6,
             ring="bf16", batch=16),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["corr", "corr", "calcorr", "calcorr", "stage1", "stage1", "imager",
                       "imager", "image", "image", "search", "search", "boxcar", "pipeline"])
    if kind == "corr":
        t_int = rng.choice([8, 16, 32])
        csf = rng.choice([4, 8, 16])
        return dict(kind=kind, n_g=rng.choice([1, 1, 2, 4]), npkt=t_int // 2 * _log(rng, 2, 120),
                    nant=16 * rng.randint(1, 6), nchan=csf * rng.randint(2, 24), t_int=t_int,
                    csf=csf, layout=rng.choice(["tbc", "tbc", "bct"]))
    if kind == "calcorr":
        t_int = rng.choice([8, 16, 32])
        csf = rng.choice([1, 2, 8, 16])
        return dict(kind=kind, npkt=t_int // 2 * _log(rng, 2, 64), nant=rng.randint(8, 96),
                    nchan=csf * rng.randint(2, 384 // csf), t_int=t_int, csf=csf,
                    dtype=rng.choice(["f16", "f16", "f32"]), fuse=rng.random() < 0.7)
    if kind == "stage1":
        return dict(kind=kind, nant=rng.randint(12, 96), n_fv=_log(rng, 64, 512),
                    chgroup=rng.randint(0, 15), csf=rng.choice([16, 32, 48]), t_int=8,
                    n_coarse=_log(rng, 3, 32), dm_max=float(rng.randint(20, 300)),
                    n_grid=rng.choice([64, 128, 256]))
    if kind == "imager":
        n = rng.choice([64, 128, 256])
        return dict(kind=kind, compact=rng.random() < 0.5, n_grid=n, n_g=rng.randint(2, 16),
                    t_det=_log(rng, 12, 64), n_fdm=rng.randint(2, 8),
                    cube=rng.choice(["f16", "f16", "f32"]), fill=_log(rng, 100, n * n // 16))
    if kind == "image":
        return dict(kind=kind, n_grid=rng.choice([64, 256, 256, 512, 512]),
                    nant=rng.randint(16, 96), n_chgroup=rng.choice([2, 4, 8]),
                    t_int=rng.choice([8, 32]), ring=rng.choice(["c64", "bf16", "cint8"]),
                    dm_max=float(rng.randint(20, 100)), n_f=rng.randint(1, 16),
                    n_t=_log(rng, 8, 144))
    if kind == "search":
        n = rng.choice([64, 128, 256, 512])
        return dict(kind=kind, n_grid=n, n_f=rng.randint(1, 8), n_out=_log(rng, 40, 256),
                    logw=rng.randint(2, 6))
    if kind == "boxcar":
        n_out = _log(rng, 16, 128)
        logw = rng.randint(1, 5)
        return dict(kind=kind, n_grid=rng.choice([64, 100, 128, 255, 256]), n_f=rng.randint(1, 4),
                    n_t=n_out + (1 << logw), n_out=n_out, logw=logw,
                    cube=rng.choice(["f16", "f32"]))
    return dict(kind=kind, n_grid=rng.choice([64, 256]), nant=16 * rng.randint(1, 4),
                n_chgroup=rng.choice([2, 4]), nchan=128, csf=rng.choice([4, 8]), t_int=8,
                npkt=1024, chunk=256, n_coarse=rng.choice([24, 32]), fine=rng.choice([1, 2]),
                dm_max=float(rng.randint(100, 400)), logw=rng.randint(2, 4),
                ring=rng.choice(["c64", "bf16", "cint8"]), batch=rng.choice([8, 12]))


# ---------------------------------------------------------------------------
# what the program has in hand
# ---------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _codes(shape, g):
    """4-bit two's-complement Gaussian voltages (sigma 3), one byte per complex
    sample, low nibble real."""
    out = torch.empty(shape, dtype=torch.uint8, device=DEV)
    flat = out.view(-1)
    for i in range(0, flat.numel(), 1 << 27):
        part = flat[i:i + (1 << 27)]
        q = [torch.randn(part.numel(), generator=g, device=DEV).mul_(3).round_().clamp_(-8, 7)
             .to(torch.int8) & 15 for _ in range(2)]
        part.copy_((q[0] | (q[1] << 4)).view(torch.uint8))
    return out


def _randn(shape, g, dtype=torch.float32):
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype)


def _gains(c, g):
    """Unit-modulus-ish antenna gains, (nchan, 1, 2, 1, nant)."""
    shape = (c["nchan"], 1, 2, 1, c["nant"])
    ph = 6.2831853 * torch.rand(shape, generator=g, device=DEV)
    amp = 1 + 0.1 * _randn(shape, g)
    dt = _DT[c["dtype"]]
    return (amp * torch.cos(ph)).to(dt), (amp * torch.sin(ph)).to(dt)


_DT = {"f16": torch.float16, "f32": torch.float32}


def _stage1(c):
    e, n = synth.t_layout(c["nant"], 17)
    cell = grid.compute_top_of_band_cell_lambda(e, n, n_grid=c["n_grid"])
    pat = grid.build_pattern(e, n, chgroup=c["chgroup"], n_grid=c["n_grid"],
                             chan_sum_factor=c["csf"], cell_lambda=cell, device=DEV)
    gr = grid.FastVisGridder.from_pattern(pat, e, n, device=DEV)
    plan = dedisp.DMPlan(dm_pc_cc=np.linspace(0.0, c["dm_max"], c["n_coarse"]),
                         t_int_fast_us=32.768 * c["t_int"], chan_sum_factor=c["csf"])
    return gr, plan


def _vis(c, g):
    nb = c["nant"] * (c["nant"] + 1) // 2
    return torch.complex(_randn((c["n_fv"], nb, 384 // c["csf"]), g).mul_(300).round_(),
                         _randn((c["n_fv"], nb, 384 // c["csf"]), g).mul_(300).round_())


def _imager_streams(c, g):
    """cint8 streams of n_g chgroups: (compact lut [n_g, N*N], compact streams
    [n_g, fill, t_pad, 2])."""
    N, G, T = c["n_grid"], c["n_g"], c["t_det"] + 16
    lut = torch.full((G, N * N), -1, dtype=torch.int64, device=DEV)
    for k in range(G):
        cells = torch.randperm(N * N, generator=g, device=DEV)[:c["fill"]].sort().values
        lut[k, cells] = torch.arange(c["fill"], device=DEV)
    q = _randn((G, c["fill"], T, 2), g).mul_(35).round_().clamp_(-127, 127).to(torch.int8)
    return lut, q


def _imager_dense(c, lut, q):
    N, G, T = c["n_grid"], c["n_g"], q.shape[2]
    full = torch.zeros((G, T, 2, N * N), dtype=torch.int8, device=DEV)
    for k in range(G):
        cells = torch.nonzero(lut[k] >= 0).reshape(-1)
        full[k, :, :, cells] = q[k, lut[k, cells]].permute(1, 2, 0)
    return full.view(G, T, 2, N, N)


def _image_pipe(c, seed):
    band = Band(n_chgroup=c["n_chgroup"])
    cfg = pipeline.PipelineConfig(
        nant=c["nant"], band=band, npkt_block=c["t_int"] // 2 * 128, t_int=c["t_int"], csf=16,
        n_grid=c["n_grid"], coarse_dm=np.array([0.5, 1.0]) * c["dm_max"], fine_per_coarse=16,
        chunk_tiles=128, fdm_batch=1, ring_dtype=c["ring"], use_sky=False, cand_capacity=1 << 16,
        layer2=False)
    e, n = synth.t_layout(c["nant"], 17)
    p = pipeline.SearchPipeline(cfg, e, n, device=DEV)
    g = _gen(seed)
    if c["ring"] == "cint8":
        p.D.view(torch.int8).copy_(_randn((p.D.numel() * 2,), g).mul_(35).round_()
                                   .clamp_(-127, 127).to(torch.int8))
        p.scales.copy_(2.0 + torch.rand(p.scales.shape, generator=g, device=DEV))
    else:
        v = _randn((p.D.numel(), 2), g).mul_(250).round_()
        p.amax.fill_(float(v.abs().max()))
        if c["ring"] == "bf16":
            p.D.copy_(v.to(torch.bfloat16).view(torch.int32).reshape(-1))
        else:
            p.D.copy_(torch.view_as_complex(v))
    return p


def _search_state(c, seed):
    N, F, C = c["n_grid"], c["n_f"], c["n_out"]
    te = (1 << c["logw"]) // 2
    g = _gen(seed)
    img = _randn((F, C + 2 * te, N, N), g)
    img *= (0.02 * (1 + 0.2 * torch.arange(F, device=DEV)))[:, None, None, None]
    # a burst of half the widest boxcar in every fine DM
    t, w = te + C // 3, max(1, te)
    for f in range(F):
        img[f, t:t + w, N // 3 + f, N // 2 + 5] += 0.3 * (1 + 0.2 * f)
    mask = torch.from_numpy(search.compute_edge_mask(n_grid=N, kernel_support=1)).to(DEV)
    act = np.nonzero(mask.reshape(-1).cpu().numpy() != 0)[0]
    pix = torch.from_numpy(act[np.linspace(0, act.size - 1, 256).astype(np.int64)]
                           .astype(np.int32)).to(DEV)
    times = torch.from_numpy((te + np.linspace(0, C - 1, 16).astype(np.int64))
                             .astype(np.int32)).to(DEV)
    K = c["logw"] + 1
    return dict(img=img, mask=mask, pix=pix, times=times, te=te,
                sinv=torch.tensor([2.0 ** (-0.5 * k) for k in range(K)], device=DEV),
                cands=search.CandidateBuffer(DEV, 1 << 20),
                l2=search.Layer2Samples(n_kernels=K, m=4096, n_out=C, n_fdm=F, npix=N * N,
                                        active=mask.cpu().numpy().reshape(-1) != 0, device=DEV))


def _boxcar_cube(c, g):
    return _randn((c["n_t"], c["n_f"], c["n_grid"], c["n_grid"]), g).to(_DT[c["cube"]])


def _pipeline_state(c, seed):
    band = DSA110_BAND if c["n_chgroup"] == 16 else \
        band_from_edges(c["n_chgroup"], c["nchan"], 1.49875, 1.31125)
    e, n = synth.t_layout(c["nant"], 17)
    cfg = pipeline.PipelineConfig(
        nant=c["nant"], band=band, npkt_block=c["npkt"], t_int=c["t_int"], csf=c["csf"],
        n_grid=c["n_grid"], coarse_dm=np.linspace(0.0, c["dm_max"], c["n_coarse"]),
        fine_per_coarse=c["fine"], log_max_width=c["logw"], threshold=7.0, sky_window=2,
        sky_warmup=1, chunk_tiles=c["chunk"], fdm_batch=c["batch"], ring_dtype=c["ring"],
        cand_capacity=1 << 22)
    p = pipeline.SearchPipeline(cfg, e, n, device=DEV)
    noise = _codes((band.n_chgroup, c["npkt"], c["nant"], band.nchan, 2, 2), _gen(seed))
    # a burst of S/N some tens, four tiles wide, that reaches the bottom of the
    # band inside the first detector cube
    dm, width = 0.4 * c["dm_max"], 4 * c["t_int"]
    nu = band.freq_table()
    late = 4.148808e3 * dm * (nu.min() ** -2 - nu[0, 0] ** -2) / 32.768
    snr = 20 * (band.n_chgroup * band.nchan / 256) ** 0.5 * (c["nant"] / 16) * (width / 4) ** 0.5
    burst = synth.Burst(dm=dm, t0_native=int((p.jc_first * c["chunk"] + 40) * c["t_int"] - late),
                        width_native=width, amp=2 * (4 / snr) ** 0.5, dl=5, dm_pix=-9)

    def block():
        raw = noise.clone()
        synth.inject_bursts_device(raw, band=band, nant=c["nant"],
                                   s0=p.chunk * c["chunk"] * c["t_int"], antpos_e=e, antpos_n=n,
                                   cell_lambda=p.tab.cell_lambda, n_grid=c["n_grid"], seed=seed,
                                   bursts=[burst])
        return raw

    # the blocks before the first detector cube fill the rings
    while p.chunk - p.depth1 - p.a < p.jc_first:
        p.process_block(block())
    raw = block()
    return dict(pipe=p, raw=raw)


def prepare(case, seed):
    c, g = case, _gen(seed)
    k = c["kind"]
    if k == "corr":
        raw = _codes((c["n_g"], c["npkt"], c["nant"], c["nchan"], 2, 2), g)
        return dict(c=c, raw=raw, k=corr.FastCorrKernel(DEV, t_int_fast_native=c["t_int"],
                                                        nants=c["nant"], nchan=c["nchan"]))
    if k == "calcorr":
        raw = _codes((c["npkt"], c["nant"], c["nchan"], 2, 2), g)
        return dict(c=c, raw=raw, gains=_gains(c, g),
                    k=corr.FastCorrKernel(DEV, t_int_fast_native=c["t_int"], nants=c["nant"],
                                          nchan=c["nchan"]))
    if k == "stage1":
        gr, plan = _stage1(c)
        st = dedisp.Stage1MultiDMCoarseDM(plan=plan, gridder=gr, chgroup=c["chgroup"],
                                          sliding_window=True)
        st.dedisperse_from_vis(_vis(c, g), block_n=0)
        return dict(c=c, st=st, vis=_vis(c, g))
    if k == "imager":
        lut, q = _imager_streams(c, g)
        sh = torch.randint(-6, 10, (c["n_fdm"], c["n_g"]), generator=g, device=DEV,
                           dtype=torch.int32)
        im = search.GpuImager.build(search.GpuImagerConfig(
            n_grid=c["n_grid"], t_det=c["t_det"], n_fdm=c["n_fdm"], n_chgroup=c["n_g"],
            cube_dtype=_DT[c["cube"]], device=DEV))
        if c["compact"]:
            kw = dict(streams_cint8=q, compact_inv_lut=lut, compact_t_stream=q.shape[2])
        else:
            kw = dict(streams_cint8=_imager_dense(c, lut, q))
        return dict(c=c, im=im, kw=dict(kw, time_shifts_gpu=sh))
    if k == "image":
        out = torch.empty((c["n_f"], c["n_t"], c["n_grid"], c["n_grid"]), device=DEV)
        return dict(c=c, pipe=_image_pipe(c, seed), out=out)
    if k == "search":
        return dict(_search_state(c, seed), c=c)
    if k == "boxcar":
        W = [1 << i for i in range(c["logw"] + 1)]
        i32 = dict(dtype=torch.int32, device=DEV)
        return dict(c=c, cube=_boxcar_cube(c, g), w=torch.tensor(W, **i32),
                    off=torch.tensor([W[-1] // 2 - w // 2 for w in W], **i32),
                    sinv=torch.tensor([w ** -0.5 for w in W], device=DEV))
    return dict(_pipeline_state(c, seed), c=c)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _rows(cols, n, dtype=np.int64):
    """The columns as n rows, those past the end -1."""
    a = np.array(cols, dtype).T
    return np.concatenate([a, np.full((n - a.shape[0], a.shape[1]), -1, a.dtype)])


SCALE = 0.05        # the voltage per 4-bit code of unpack_int4_split's default


def run(state):
    s, c = state, state["c"]
    k = c["kind"]
    if k == "corr":
        return s["k"].compute_raw(s["raw"], chan_sum_factor=c["csf"], layout=c["layout"])
    if k == "calcorr":
        re, im = corr.unpack_int4_split(s["raw"], device=DEV, scale=SCALE,
                                        out_dtype=_DT[c["dtype"]], npkt=c["npkt"],
                                        nant=c["nant"], nchan=c["nchan"])
        re, im = corr.apply_cal_split(re, im, *s["gains"])
        return s["k"].compute_split(re, im, fuse_stokes_i=c["fuse"],
                                    chan_sum_factor=c["csf"] if c["fuse"] else 1)
    if k == "stage1":
        return s["st"].dedisperse_from_vis(s["vis"], block_n=1)
    if k == "imager":
        return s["im"].process_cube(**s["kw"])
    if k == "image":
        s["pipe"].image(0, c["n_f"], 700, c["n_t"], s["out"])
        return s["out"]
    if k == "search":
        sig = search.layer1_sigma(s["img"], s["times"], s["pix"])
        s["cands"].reset()
        search.detect_images(s["img"], s["mask"], log_max_width=c["logw"], sigma_inv=s["sinv"],
                             t_base=s["te"], n_out=c["n_out"], threshold=7.0, cands=s["cands"],
                             sigma_f=sig, layer2=s["l2"])
        sk = search.sigma_clipped_std_batched(s["l2"].samples)
        n_top = 64 * (c["logw"] + 1)
        got = s["cands"].fetch_top(n_top)
        got = got[np.lexsort((got["pix"], got["t"], -got["snr"]))][:n_top]
        return dict(sigma=sig, samples=s["l2"].samples, sigma_k=sk,
                    cands=_rows([got["t"], got["pix"], got["k"]], n_top),
                    snr=_rows([got["snr"]], n_top, np.float32))
    if k == "boxcar":
        cs = search.precompute_padded_cumsum(s["cube"], axis=0, max_width=1 << c["logw"])
        return search.multi_boxcar_argmax_triton(
            cs, widths=s["w"], offsets=s["off"], sigma_inv=s["sinv"], n_out=c["n_out"],
            t_base=(1 << c["logw"]) // 2)
    p = s["pipe"]
    got = p.process_block(s["raw"])[:64]
    cands = [[getattr(q, f) for q in got] for f in ("t", "fdm", "l", "m", "width")]
    return dict(cands=_rows(cands, 64), snr=_rows([[q.snr for q in got]], 64, np.float32),
                ring=p.D, images=p.img)


def work(case):
    """Bytes that one pass reads and writes once, and its operations."""
    c = case
    k = c["kind"]
    if k in ("corr", "calcorr"):
        samp = c.get("n_g", 1) * c["npkt"] * c["nant"] * c["nchan"] * 4
        nb = c["nant"] * (c["nant"] + 1) // 2
        n_fv = c["npkt"] * 2 // c["t_int"]
        n_out = c["nchan"] // c["csf"] if c.get("fuse", True) else 2 * c["nchan"]
        return dict(bytes=samp + c.get("n_g", 1) * n_fv * nb * n_out * 8,
                    flops=8 * nb * samp // c["nant"])
    if k == "stage1":
        nb = c["nant"] * (c["nant"] + 1) // 2
        src = nb * (384 // c["csf"])
        cells = min(nb, c["n_grid"] ** 2 // 2)
        return dict(bytes=2 * c["n_fv"] * src * 8 + c["n_coarse"] * c["n_fv"] * cells * 8,
                    flops=2 * c["n_coarse"] * c["n_fv"] * src)
    if k == "imager":
        N = c["n_grid"]
        px = c["t_det"] * c["n_fdm"] * N * N
        cells = c["fill"] if c["compact"] else N * N
        return dict(bytes=c["n_g"] * (c["t_det"] + 16) * cells * 2 +
                    px * (2 if c["cube"] == "f16" else 4),
                    flops=px * 5 * int(np.log2(N)))
    if k == "image":
        N = c["n_grid"]
        px = c["n_f"] * c["n_t"] * N * N
        cells = min(c["nant"] * (c["nant"] + 1) // 2, N * N // 2) * c["n_chgroup"]
        el = {"c64": 8, "bf16": 4, "cint8": 2}[c["ring"]]
        return dict(bytes=px * 4 + (c["n_t"] + 16) * cells * el, flops=px * 5 * int(np.log2(N)))
    if k == "search":
        px = c["n_f"] * (c["n_out"] + (1 << c["logw"])) * c["n_grid"] ** 2
        return dict(bytes=px * 4, flops=px * (c["logw"] + 2))
    if k == "boxcar":
        inner = c["n_f"] * c["n_grid"] ** 2
        return dict(bytes=c["n_t"] * inner * (2 if c["cube"] == "f16" else 4) +
                    c["n_out"] * inner * 6, flops=c["n_out"] * inner * 2 * (c["logw"] + 1))
    samp = c["n_chgroup"] * c["npkt"] * c["nant"] * c["nchan"] * 4
    px = c["n_coarse"] * c["fine"] * (c["chunk"] + (1 << c["logw"])) * c["n_grid"] ** 2
    return dict(bytes=samp + 8 * px, flops=px * (5 * int(np.log2(c["n_grid"])) + c["logw"] + 2)
                + 4 * (c["nant"] + 1) * samp)


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------

def _decode(raw):
    """On-wire bytes -> complex128 codes."""
    lo, hi = (raw & 15).to(torch.int16), (raw >> 4).to(torch.int16)
    return torch.complex((lo - 16 * (lo > 7)).double(), (hi - 16 * (hi > 7)).double())


def _xcorr(c, raw, gains=None, fuse=True):
    """(n_fv, nbase, nchan / csf) or (n_fv, nbase, nchan, 2) of one page."""
    na, csf = c["nant"], c["csf"] if fuse else 1
    pp = c["t_int"] // 2
    n_fv = c["npkt"] // pp
    a, b = torch.tril_indices(na, na, device=DEV)
    outs = []
    for ch in range(0, c["nchan"], csf):
        v = _decode(raw[:, :, ch:ch + csf]).view(n_fv, pp, na, csf, 2, 2)
        if gains is not None:
            gn = torch.complex(gains[0][ch:ch + csf].double(), gains[1][ch:ch + csf].double())
            v = v * SCALE * gn[:, 0, :, 0].permute(2, 0, 1)[None, None, :, :, None, :]
        v = v.permute(5, 0, 1, 3, 4, 2).reshape(2, n_fv, pp * csf * 2, na)   # (pol, f, k, ant)
        m = v.transpose(2, 3) @ v.conj()                                     # E_a conj(E_b)
        m = m[:, :, a, b]
        outs.append(m.sum(0) if fuse else m.permute(1, 2, 0))
    return torch.stack(outs, 2)


def _half_to_image(half, N):
    u, w = torch.arange(N, device=DEV)[:, None], torch.arange(N // 2 + 1, device=DEV)[None]
    return torch.fft.irfft2(half * (1 - 2 * ((u + w) & 1)), s=(N, N))


def _clipped_std(rows):
    out = []
    for r in rows.double():
        act = r[torch.isfinite(r)]
        for it in range(4):
            med = act.sort().values[(act.numel() - 1) // 2]
            sig = ((act - med) ** 2).mean().sqrt()
            if it < 3:
                act = act[(act >= med - 3 * sig) & (act <= med + 3 * sig)]
        out.append(sig)
    return torch.stack(out)


def exact(case, seed):
    c = case
    k = c["kind"]
    N = c.get("n_grid")
    if k == "pipeline":
        return None
    s = prepare(case, seed)
    if k == "corr":
        v = torch.stack([_xcorr(c, r) for r in s["raw"]])
        return v.permute(0, 2, 3, 1) if c["layout"] == "bct" else v
    if k == "calcorr":
        return _xcorr(c, s["raw"], s["gains"], c["fuse"])
    if k == "stage1":
        g = _gen(seed)
        v = torch.cat([_vis(c, g), _vis(c, g)])
        st = s["st"]
        cim = st.gridder.cell_index_map.view(v.shape[1], v.shape[2]).to(DEV)
        sh = st.plan.delay_bins_per_chgroup(c["chgroup"])
        out = torch.zeros((c["n_coarse"], c["n_fv"], st.n_filled_out + 1, 2),
                          dtype=torch.float64, device=DEV)
        for d in range(c["n_coarse"]):
            for ch in range(v.shape[2]):
                x = v[sh[ch, d]:sh[ch, d] + c["n_fv"], :, ch].to(torch.complex128)
                out[d].index_add_(1, cim[:, ch], torch.view_as_real(x.contiguous()))
        return torch.view_as_complex(out[:, :, :-1].contiguous())
    if k == "imager":
        q = s["kw"]["streams_cint8"]
        if c["compact"]:
            q = _imager_dense(c, s["kw"]["compact_inv_lut"], q)
        idx = (-torch.arange(N, device=DEV)) % N
        pad = 4                     # kernel_support 5: 5 // 2 + 2
        mask = torch.zeros((N, N), dtype=torch.float64, device=DEV)
        mask[pad:N - pad, pad:N - pad] = 1
        mask[N // 2, N // 2] = 0
        i = torch.arange(N, device=DEV)
        mask *= 1 - 2 * ((i[:, None] + i[None]) & 1)
        sh = s["kw"]["time_shifts_gpu"].cpu().numpy()
        cube = torch.empty((c["t_det"], c["n_fdm"], N, N), dtype=torch.float64, device=DEV)
        for f in range(c["n_fdm"]):
            for t0 in range(0, c["t_det"], 16):
                t = torch.arange(t0, min(t0 + 16, c["t_det"]), device=DEV)
                z = torch.zeros((t.numel(), N, N), dtype=torch.complex128, device=DEV)
                for j in range(c["n_g"]):
                    ts = t - int(sh[f, j])
                    ok = (ts >= 0) & (ts < q.shape[1])
                    x = q[j, ts.clamp(0, q.shape[1] - 1)].double() * ok[:, None, None, None]
                    z += torch.complex(x[:, 0], x[:, 1])
                half = 0.5 * (z + z[:, idx][:, :, idx].conj())[:, :, :N // 2 + 1]
                cube[t0:t0 + 16, f] = _half_to_image(half, N) * mask
        return cube
    if k == "image":
        p = s["pipe"]
        T, nh = p.tab, N // 2 + 1
        cell = torch.from_numpy(np.repeat(np.arange(N * nh), np.diff(T.hc_off))).to(DEV)
        eg = torch.from_numpy(T.e_g.astype(np.int64)).to(DEV)
        ec = torch.from_numpy(T.e_cell.astype(np.int64)).to(DEV)
        conj = ec < 0
        ec = torch.where(conj, -1 - ec, ec)
        out = torch.empty(s["out"].shape, dtype=torch.float64, device=DEV)
        nc = p.cfg.coarse_dm.size
        for f in range(c["n_f"]):
            gc = np.arange(c["n_chgroup"]) * nc + int(p.cfg.fine_to_coarse[f])
            for t in range(c["n_t"]):
                slot = (700 + t - T.sfine[f].astype(np.int64)) % p.seg_depth[gc]
                base = torch.from_numpy(p.seg_base[:-1][gc] + slot * T.pitch).to(DEV)
                v = p.D[base[eg] + ec]
                if c["ring"] == "c64":
                    v = torch.view_as_real(v).double()
                elif c["ring"] == "bf16":
                    v = v.view(torch.bfloat16).view(-1, 2).double()
                else:
                    sc = p.scales[torch.from_numpy(p.sc_base[:-1][gc] + slot).to(DEV)].double()
                    v = v.view(torch.int8).view(-1, 2).double() * sc[eg][:, None]
                v[:, 1] *= 1 - 2 * conj.double()
                h = torch.zeros((N * nh, 2), dtype=torch.float64, device=DEV)
                h.index_add_(0, cell, v)
                out[f, t] = _half_to_image(0.5 * torch.view_as_complex(h).view(N, nh), N)
        return out
    if k == "search":
        img, te = s["img"], s["te"]
        F = c["n_f"]
        samp = img.view(F, img.shape[1], -1)[:, s["times"].long()][:, :, s["pix"].long()]
        sig = _clipped_std(samp.reshape(F, -1))
        got = torch.full(s["l2"].samples.shape, float("nan"), dtype=torch.float64, device=DEV)
        ent = torch.from_numpy(s["l2"].entries).to(DEV)
        for i in range(c["logw"] + 1):
            e = ent[ent[:, 2] == i]
            f, p = e[:, 0] // (N * N), e[:, 0] % (N * N)
            lo = te + e[:, 1] - (1 << i) // 2
            x = torch.zeros(e.shape[0], dtype=torch.float64, device=DEV)
            for j in range(1 << i):
                t = lo + j
                ok = (t >= 0) & (t < img.shape[1])
                x += img[f, t.clamp(0, img.shape[1] - 1), p // N, p % N].double() * ok
            got[i, e[:, 3]] = x * s["mask"].view(-1)[p].double() / sig[f]
        return dict(sigma=sig, samples=got, sigma_k=_clipped_std(got), cands=None, snr=None)
    cs = torch.zeros((c["n_t"] + 2 * (1 << c["logw"]),) + s["cube"].shape[1:],
                     dtype=torch.float64, device=DEV)
    h = (1 << c["logw"]) // 2
    cs[1 + h:1 + h + c["n_t"]] = s["cube"].double().cumsum(0)
    cs[1 + h + c["n_t"]:] = cs[h + c["n_t"]]
    best = None
    for w, off, si in zip(s["w"].tolist(), s["off"].tolist(), s["sinv"].double().tolist()):
        x = (cs[h + off + w:h + off + w + c["n_out"]] - cs[h + off:h + off + c["n_out"]]) * si
        best = x if best is None else torch.maximum(best, x)
    return best, None
