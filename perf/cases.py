"""Timed cases of the two-stage direct-sum pipeline.

Four kinds of work that a user of the library has it do:

  day    one whole day on a resident sky (`Pipeline.run`): stage 1 and stage 2 of every segment;
  host   one whole day from host memory to host memory (`Pipeline.run_host`), as the drop-in executables run it;
  viss   the stage-1 sum of one segment or sky slab through the C ABI (`vb_viss_halfsym`, then
         `vb_phase_correct_expand` to the float32 visibilities that the files and stage 2 take);
  image  the stage-2 reconstruction of given visibilities through the C ABI (`vb_recon_batched`).

A case names the sky (nside, and for viss / image a range of NEST pixels), the formation ("lunar": the
upstream's eight trailing satellites on a lunar orbit, sampled at its own step; "earth": satellites on
circular orbits at 400-600 km, `dt_s` seconds a step), the wavelength, the number of steps, and the options
of the call.  The sky is U[0,1) plus 20 point sources of amplitude 10, the orbit phases come from the seed.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import viss_optimize_ws_b200 as vb
from viss_optimize_ws_b200.sharded import DeviceView

LUNAR = dict(orbit="lunar", nsat=8, dt_s=0.0)
PRECISIONS = {"ref32": 0, "fp64": 1, "fp32_fp64phase": 2, "fp32_dsphase": 3}
CULLS = {"none": 0, "tilecone": 1, "exact": 2}


def _day(name, **kw):
    d = dict(name=name, kind="day", nside=64, orbit="earth", nsat=8, dt_s=2.0, steps=64, segs=4, lam=30.0, cull="tilecone",
             tile_pix=1024, mirror=1, occ_mode=2, blockage=1, grid_res=0, precision="fp32_fp64phase", uneven=0, day=1)
    return dict(d, **kw)


def _viss(name, **kw):
    d = dict(name=name, kind="viss", nside=64, base=0, npix=49152, orbit="lunar", nsat=8, dt_s=0.0, steps=64, lam=300.0, day=1,
             cull="tilecone", tile_pix=256, blockage=1, corrected=1, precision="fp32_fp64phase")
    return dict(d, **kw)


def _image(name, **kw):
    d = dict(name=name, kind="image", nside=64, base=0, npix=49152, orbit="lunar", nsat=8, dt_s=0.0, steps=64, segs=1, lam=300.0,
             day=1, mirror=1, occ_mode=2, blockage=1, cull="exact", grid_res=0, precision="fp32_fp64phase")
    return dict(d, **kw)


def listed():
    return [
        # a short segment on a coarse sky: the smallest call in use, where launches and latency count
        _viss("segment_small", nside=32, npix=12288, steps=40, tile_pix=256),
        # the size the plain method runs on host cores: no tile culling, the full signed grid
        _day("day_nside64_plain", nside=64, steps=64, segs=4, cull="none", mirror=0, grid_res=256),
        # a sky slab that is a multiple of nothing, 7 satellites, the upstream kernel's raw phase, exact culling
        _viss("slab_odd_raw", nside=128, base=40961, npix=100003, orbit="earth", nsat=7, dt_s=3.0, steps=333, lam=30.0, cull="exact",
              corrected=0),
        # the second configuration of the benchmark: 10 MHz, nside 256, 512 x 512 mirrored grid
        _day("day_nside256_10MHz", nside=256, steps=1024, segs=4, grid_res=513),
        # many short segments of uneven length in one batch
        _day("day_64_uneven_segments", nside=256, steps=0, segs=64, uneven=1, grid_res=512),
        # a 30 MHz day of 12 satellites: the longest baselines (|u| to 1e5 wavelengths)
        _day("day_nside512_30MHz", nside=512, nsat=12, steps=1000, segs=16, lam=10.0, tile_pix=4096, grid_res=512),
        # the upstream's own 1 MHz setting: lunar formation, ten segments, 256-pixel tiles, its default grid
        _day("day_1MHz_lunar", **LUNAR, nside=512, steps=0, segs=10, lam=300.0, tile_pix=256),
        # the root executable's settings from host memory: no tile cones, the full signed grid, a later day of the formation
        _day("host_day_1MHz_full_grid", kind="host", **LUNAR, nside=128, steps=0, segs=10, lam=300.0, cull="none", mirror=0, day=5),
        # the largest single-GPU day: nside 1024, 120 baselines, 128 segments
        _day("day_nside1024_128_segments", nside=1024, nsat=16, steps=2048, segs=128, lam=300.0, tile_pix=16384, grid_res=1024),
        # part of a segment of the upstream's 10 MHz production day on a fine sky
        _viss("segment_10MHz_lunar", nside=1024, npix=12582912, steps=997, lam=30.0, day=3),
        # reconstruction of one 10 MHz segment on part of that sky
        _image("image_10MHz_lunar", nside=512, npix=1000003, steps=2000, lam=30.0, day=3),
        # reconstruction with four sampled members a group, signed grid (occ_mode 3)
        _image("image_samples_full_grid", nside=64, npix=49152, steps=250, segs=3, mirror=0, occ_mode=3, cull="none"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    case = _draw(rng)
    del case["name"]
    return case


def _draw(rng):
    kind = rng.choice(["day", "day", "viss", "viss", "viss", "image", "image", "host"])
    nside = rng.choice([32, 64, 128, 256, 512, 1024])
    lunar = rng.random() < 0.5
    lam = rng.choice([300.0, 300.0, 30.0, 30.0, 10.0])
    o = dict(orbit="lunar", nsat=8, dt_s=0.0) if lunar else dict(orbit="earth", nsat=rng.randint(3, 16), dt_s=round(rng.uniform(0.5, 4.0), 2))
    pairs = o["nsat"] * (o["nsat"] - 1) // 2
    precision = rng.choice(["fp32_fp64phase"] * 7 + ["fp32_dsphase", "fp64", "ref32"])
    slow = {"fp64": 12, "fp32_dsphase": 3}.get(precision, 1)
    blockage = 0 if rng.random() < 0.1 else 1
    day = rng.randint(1, 14)
    if kind in ("day", "host"):
        if lunar:
            lam = 300.0   # the formation's own plan at 10 and 30 MHz has 7e4 steps and more
        steps = 0 if lunar else _log_uniform(rng, 48, 2048)
        total = 6980 if lunar else steps
        while 12 * nside * nside * pairs * total * slow > 1.5e12:
            nside //= 2
        mirror = rng.randint(0, 1) if nside <= 256 else 1
        # sampling the members of every group costs several masks a term: small skies
        occ = rng.choice([0, 1, 3]) if (not lunar and blockage and nside <= 64 and rng.random() < 0.3) else 2
        return _day("", kind=kind, nside=nside, **o, steps=steps, segs=rng.randint(1, min(64, total)), lam=lam,
                    cull=rng.choice(["tilecone", "tilecone", "exact", "none"]), tile_pix=rng.choice([256, 512, 1024, 4096]),
                    mirror=mirror, occ_mode=occ, blockage=blockage, grid_res=0 if lam == 300.0 and lunar else rng.choice([256, 513, 1024]),
                    precision=precision, day=day)
    npix = min(_log_uniform(rng, 9000, 6e6), 12 * nside * nside)
    base = rng.randint(0, 12 * nside * nside - npix)
    steps = _log_uniform(rng, 9, 2500)
    if kind == "viss":
        while npix * pairs * steps * slow > 3e11:
            steps = max(1, steps // 2)
        return _viss("", nside=nside, base=base, npix=npix, **o, steps=steps, lam=lam, day=day,
                     cull=rng.choice(["tilecone", "tilecone", "exact", "none"]), tile_pix=rng.choice([256, 512, 1024, 4096]),
                     blockage=blockage, corrected=rng.randint(0, 3) and 1, precision=precision)
    occ = rng.choice([2, 2, 2, 2, 0, 1, 3])
    slow *= 40 if occ != 2 else 1
    while npix * pairs * steps * slow > 2e11:
        steps = max(1, steps // 2)
    return _image("", nside=nside, base=base, npix=npix, **o, steps=steps, segs=rng.randint(1, min(40, steps)), lam=lam, day=day,
                  mirror=rng.randint(0, 1), occ_mode=occ, blockage=blockage, cull=rng.choice(["exact", "exact", "none"]),
                  grid_res=rng.choice([0, 513, 1024]) if lam == 300.0 else rng.choice([513, 1024]), precision=precision)


# --- inputs ---------------------------------------------------------------------
def _nest_xyz(nside, base, count):
    """Unit vectors of NEST pixels [base, base + count) in FP64 (Gorski et al. 2005)."""
    p = torch.arange(base, base + count, dtype=torch.int64, device="cuda")
    face, q = p // (nside * nside), p % (nside * nside)
    ix, iy = torch.zeros_like(q), torch.zeros_like(q)
    for b in range(nside.bit_length() - 1):
        ix |= ((q >> (2 * b)) & 1) << b
        iy |= ((q >> (2 * b + 1)) & 1) << b
    del q, p
    row = torch.tensor([2, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 4], device="cuda")[face]
    col = torch.tensor([1, 3, 5, 7, 0, 2, 4, 6, 1, 3, 5, 7], device="cuda")[face]
    jr = row * nside - ix - iy - 1
    north, south = jr < nside, jr > 3 * nside
    nr = torch.where(north, jr, torch.where(south, 4 * nside - jr, torch.full_like(jr, nside)))
    cap = (nr * nr).double() / (3.0 * nside * nside)
    z = torch.where(north, 1 - cap, torch.where(south, cap - 1, (2 * nside - jr).double() * 2 / (3.0 * nside)))
    shift = torch.where(north | south, torch.zeros_like(jr), (jr - nside) & 1)
    jp = (col * nr + ix - iy + 1 + shift) // 2
    phi = (jp.double() - 0.5 * (shift + 1)) * (math.pi / 2) / nr
    st = torch.where(north | south, torch.sqrt(cap * (2 - cap)), torch.sqrt((1 - z) * (1 + z)))
    return st * torch.cos(phi), st * torch.sin(phi), z


def _formation(case, seed):
    """Float32 satellite positions (km), [step][satellite][xyz]."""
    rng = np.random.default_rng(seed)
    steps, nsat = case["steps"], case["nsat"]
    if case["orbit"] == "lunar":
        # 2.3 h orbit sampled so that the longest baseline turns by one wavelength a step; the trailing
        # distances grow and shrink over 14 days
        per_rev = math.ceil(2 * math.pi * 100e3 / case["lam"])
        th = rng.uniform(0, 2 * math.pi) + 2 * math.pi * np.arange(steps + 1) / per_rev
        raan, incl, r = rng.uniform(0, 2 * math.pi), math.radians(30), 2038.14
        s = 100.0 / 23.0
        far = np.array([0, s, 4 * s, 10 * s, 16 * s, 18 * s, 21 * s, 23 * s])
        f = (case["day"] - 1) / 7.0
        dist = far * (0.1 + 0.9 * (f if f <= 1 else 2 - f))
        x = np.stack([np.cos(th) * math.cos(raan) - np.sin(th) * math.cos(incl) * math.sin(raan),
                      np.cos(th) * math.sin(raan) + np.sin(th) * math.cos(incl) * math.cos(raan), np.sin(th) * math.sin(incl)], -1) * r
        v = np.diff(x, axis=0)
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        return (x[1:, None, :] - dist[None, :, None] * v[:, None, :]).astype(np.float32)
    t = np.arange(steps) * case["dt_s"]
    incl0, raan0, u0 = rng.uniform(math.radians(20), math.radians(80)), rng.uniform(0, 2 * math.pi), rng.uniform(0, 2 * math.pi)
    out = np.empty((steps, nsat, 3), np.float32)
    for k in range(nsat):
        r = 6371.0 + rng.uniform(400, 600)
        a = 50.0 / r
        i, o = incl0 + a * rng.uniform(-0.5, 0.5), raan0 + a * rng.uniform(-0.5, 0.5)
        th = u0 + a * rng.uniform(-1, 1) + math.sqrt(398600.4418 / r**3) * t
        out[:, k, 0] = r * (np.cos(th) * math.cos(o) - np.sin(th) * math.cos(i) * math.sin(o))
        out[:, k, 1] = r * (np.cos(th) * math.sin(o) + np.sin(th) * math.cos(i) * math.cos(o))
        out[:, k, 2] = r * np.sin(th) * math.sin(i)
    return out


def _baselines(case, seed):
    """Signed baselines in the library's layout ([pairs "-"][pairs "+"] per step) as float32 device tensors."""
    x = _formation(case, seed)
    a, b = np.triu_indices(case["nsat"], 1)
    xa, xb = x[:, a], x[:, b]
    d = ((xb - xa) * np.float32(1e3) / np.float32(case["lam"])).astype(np.float32)
    uvw = np.concatenate([-d, d], 1).reshape(-1, 3)
    e1, e2 = np.concatenate([xb, xa], 1).reshape(-1, 3), np.concatenate([xa, xb], 1).reshape(-1, 3)
    t = {}
    for names, arr in ((("u", "v", "w"), uvw), (("x1", "y1", "z1"), e1), (("x2", "y2", "z2"), e2)):
        for k, n in enumerate(names):
            t[n] = torch.from_numpy(np.ascontiguousarray(arr[:, k])).cuda()
    for k, e in (("1", e1), ("2", e2)):
        t["invn" + k] = torch.rsqrt(t["x" + k] * t["x" + k] + t["y" + k] * t["y" + k] + t["z" + k] * t["z" + k])
        if case["orbit"] == "earth":   # the Earth's horizon seen from each endpoint
            r = np.linalg.norm(e.astype(np.float64), axis=1)
            t["cosphi" + k] = torch.from_numpy((-np.sqrt(np.maximum(0.0, 1.0 - (6371.0 / r) ** 2))).astype(np.float32)).cuda()
    # the lunar set-up's one horizon cosine (R = 1737.1 km, h = 300 km)
    t["cosphi"] = float(np.cos(np.float32(math.pi) - np.arcsin(np.float32(1737.1e3 / 2037.1e3)), dtype=np.float32))
    return t


def _sky(case, seed, scaled=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    full = 12 * case["nside"] ** 2
    n = case.get("npix", full)
    B = torch.rand(n, generator=g, device="cuda")
    B[torch.randint(n, (20,), generator=g, device="cuda")] += 10.0
    return B * np.float32(4 * math.pi / full) if scaled else B


def _segments(case):
    cuts = np.linspace(0, case["steps"], case["segs"] + 1).astype(np.int32)
    return cuts[:-1], np.diff(cuts).astype(np.int32)


def _visibilities(case, t, seed):
    """Float32 (re, im) of every half-baseline: a few sources and noise."""
    rng = np.random.default_rng(seed + 1)
    half = _half(case)
    u = torch.stack([t[k].double()[half] for k in "uvw"], 1)
    V = torch.zeros(half.numel(), dtype=torch.complex128, device="cuda")
    for _ in range(8):
        s = rng.normal(size=3)
        V += rng.uniform(0.1, 1) * torch.exp(-2j * math.pi * (u @ torch.from_numpy(s / np.linalg.norm(s)).cuda()))
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    V = torch.view_as_real(V) + 0.1 * torch.randn(half.numel(), 2, generator=g, device="cuda", dtype=torch.float64)
    return V.float().contiguous()


def _half(case):
    nbl = case["nsat"] * (case["nsat"] - 1) // 2
    i = torch.arange(nbl * case["steps"], device="cuda")
    return (i // nbl) * 2 * nbl + i % nbl


def _grid(case):
    """(bl_max, grid_res) of the uv grid: the upstream's 100 km for the lunar formation, else one that covers the tracks."""
    return (100e3 if case["orbit"] == "lunar" else 0.0), case["grid_res"]


def prepare(case, seed):
    L = vb.lib()
    if case["kind"] in ("day", "host"):
        lunar = case["orbit"] == "lunar"
        cfg = vb.run_config(nside=case["nside"], orbit_model=vb.ORBIT_REFERENCE if lunar else vb.ORBIT_SYNTHETIC, nsat=case["nsat"],
                            tsteps=case["steps"], dt_s=case["dt_s"] or 2.0, segs=case["segs"], seg_plan=case["uneven"],
                            lambda_m=case["lam"], occ_R_m=0.0 if lunar else 6371e3, cull=case["cull"], viss_tile_pix=case["tile_pix"],
                            mirror=case["mirror"], occ_mode=case["occ_mode"], blockage=case["blockage"], grid_res=case["grid_res"],
                            bl_max_m=_grid(case)[0], orbit_seed=seed, day=case["day"], precision=case["precision"])
        p = vb.Pipeline(cfg)
        B = _sky(case, seed, scaled=False).cpu().numpy()
        if case["kind"] == "host":
            return {"case": case, "p": p, "B": B}
        p.set_sky(B)
        p.make_baselines()
        out = {}
        for name, dt in (("C", np.float32), ("W", np.int32), ("V_half", np.float32)):
            ptr, n = p.ptr(name)
            view = DeviceView(ptr, n, dt)
            view.owner = p   # the tensor keeps the view, and so the pipeline whose buffer it is
            out[name] = view.tensor("cuda")
        return {"case": case, "p": p, "out": out}

    l, m, n = (a.float().contiguous() for a in _nest_xyz(case["nside"], case["base"], case["npix"]))
    t = _baselines(case, seed)
    st = {"case": case, "l": l, "m": m, "n": n, "B": _sky(case, seed), "t": t}
    sky = vb.Sky(npix=case["npix"], B=st["B"].data_ptr(), l=l.data_ptr(), m=m.data_ptr(), n=n.data_ptr())
    nbl = case["nsat"] * (case["nsat"] - 1) // 2
    bl = vb.Baselines(n_full=2 * nbl * case["steps"], nbl=nbl, cosphi=t["cosphi"])
    for k, v in t.items():
        if k != "cosphi":
            setattr(bl, k, v.data_ptr())
    st["sky"], st["bl"] = sky, bl
    n_half = bl.n_full // 2
    if case["kind"] == "viss":
        if case["cull"] == "tilecone":
            tiles = -(-case["npix"] // case["tile_pix"])
            st["tiles"] = torch.zeros(5, tiles, device="cuda")
            cone = [st["tiles"][k].data_ptr() for k in range(5)]
            torch.cuda.synchronize()
            vb.check(L.vb_tile_cone_meta(case["tile_pix"], l.data_ptr(), m.data_ptr(), n.data_ptr(), case["npix"], *cone, None))
            sky.tile_pix = case["tile_pix"]
            sky.cx, sky.cy, sky.cz, sky.cosA, sky.sinA = cone
        st["opts"] = vb.Stage1Opts(precision=PRECISIONS[case["precision"]], cull=CULLS[case["cull"]],
                                   phase_corrected=case["corrected"], blockage=case["blockage"])
        need = L.vb_stage1_workspace_bytes(C.byref(sky), C.byref(bl), C.byref(st["opts"]))
        st["V"] = torch.zeros(2 * n_half, dtype=torch.float64, device="cuda")
        st["Vh"] = torch.zeros(2 * n_half, device="cuda")
    else:
        st["V"] = _visibilities(case, t, seed)
        t0, tl = _segments(case)
        st["t0"], st["tl"] = torch.from_numpy(t0).cuda(), torch.from_numpy(tl).cuda()
        st["opts"] = vb.Stage2Opts(mirror=case["mirror"], blockage=case["blockage"], occ_mode=case["occ_mode"],
                                   precision=PRECISIONS[case["precision"]], cull=CULLS[case["cull"]], grid_res=case["grid_res"],
                                   bl_max=_bl_max(case, t), lambda_=case["lam"])
        need = L.vb_stage2_workspace_bytes(n_half, case["segs"], case["npix"], C.byref(st["opts"]))
        st["C"] = torch.zeros(case["npix"], device="cuda")
        st["W"] = torch.zeros(case["npix"], dtype=torch.int32, device="cuda")
    if not need:
        raise RuntimeError(L.vb_last_error().decode())
    st["ws"] = torch.zeros(need, dtype=torch.uint8, device="cuda")
    return st


def _bl_max(case, t):
    fixed = _grid(case)[0]
    return fixed or float(np.float32(float(max(t["u"].abs().max(), t["v"].abs().max())) * case["lam"] * 1.0001))


def run(state):
    kind = state["case"]["kind"]
    if kind == "day":
        state["p"].run()
        return state["out"]
    if kind == "host":
        image, V, _ = state["p"].run_host(state["B"], want_v=True)
        return {"C": image, "V_half": V}
    L, s, ws = vb.lib(), torch.cuda.current_stream().cuda_stream, state["ws"]
    sky, bl, o = C.byref(state["sky"]), state["bl"], C.byref(state["opts"])
    if kind == "viss":
        vb.check(L.vb_viss_halfsym(sky, C.byref(bl), o, ws.data_ptr(), ws.numel(), state["V"].data_ptr(), None, s))
        vb.check(L.vb_phase_correct_expand(state["V"].data_ptr(), state["t"]["w"].data_ptr(), bl.n_full // 2, bl.nbl,
                                           state["case"]["corrected"], state["Vh"].data_ptr(), None, s))
        return {"V_half": state["Vh"]}
    vb.check(L.vb_recon_batched(sky, C.byref(bl), state["V"].data_ptr(), state["case"]["segs"], state["t0"].data_ptr(),
                                state["tl"].data_ptr(), o, ws.data_ptr(), ws.numel(), state["C"].data_ptr(), state["W"].data_ptr(),
                                None, None, s))
    return {"C": state["C"], "W": state["W"]}


# --- work and 64-bit values --------------------------------------------------------
def _sizes(case):
    """(pixels, half-baselines, uv groups): the groups as an estimate, 0.3 a half-baseline."""
    npix = case.get("npix", 12 * case["nside"] ** 2)
    pairs = case["nsat"] * (case["nsat"] - 1) // 2
    steps = case["steps"]
    if not steps:
        steps = case["segs"] * 1025 // pairs if case["uneven"] else 10 * (math.ceil(2 * math.pi * 100e3 / case["lam"]) // 3)
    return npix, pairs * steps, max(1, int(0.3 * pairs * steps))


def work(case):
    """Ten operations a visible (pixel, baseline) or (pixel, group) pair -- three multiply-adds of phase, a sine and a cosine, two
    multiply-adds -- of which the occluder leaves about 0.7; sky and image, baselines and visibilities once."""
    npix, half, groups = _sizes(case)
    both = case["kind"] in ("day", "host")
    pairs = npix * ((half if both or case["kind"] == "viss" else 0) + (groups if both or case["kind"] == "image" else 0))
    seen = 0.7 if case["blockage"] else 1.0
    return {"bytes": 16 * npix + (8 * npix if case["kind"] != "viss" else 0) + 2 * half * 44 + 8 * half, "flops": 12 * seen * pairs}


def _fma(a, b, c):
    """fl(a b + c) of float32 tensors (a product of two floats is exact in a double)."""
    return (a.double() * b.double() + c.double()).float()


def _seen(sky, t, idx):
    """The occlusion test of both endpoints as the kernels' float32 steps decide it, [pixel][baseline]."""
    ok = None
    for k in ("1", "2"):
        x, y, z, i = (t[c + k][idx][None, :] for c in ("x", "y", "z", "invn"))
        l, m, n = (a[:, None] for a in sky)
        d = _fma(n, z, _fma(l, x, m * y)) * i
        c = t["cosphi" + k][idx][None, :] if "cosphi" + k in t else np.float32(t["cosphi"])
        ok = d >= c if ok is None else ok & (d >= c)
    return ok


def exact(case, seed):
    npix, half, groups = _sizes(case)
    if case["kind"] in ("day", "host"):
        return None   # the float32 orbit tables are the library's own
    if case["kind"] == "viss":
        if npix * half > 2.5e10:
            return None
        return {"V_half": _exact_viss(case, seed)}
    if case["blockage"] and case["occ_mode"] != 2 or npix * groups > 2.5e10:
        return None
    return _exact_image(case, seed)


def _exact_viss(case, seed):
    xyz = [a.float() for a in _nest_xyz(case["nside"], case["base"], case["npix"])]
    t, B = _baselines(case, seed), _sky(case, seed).double()
    half = _half(case)
    S = torch.stack([a.double() for a in xyz], 1)
    U = torch.stack([t[k].double()[half] for k in "uvw"], 1)
    V = torch.zeros(half.numel(), 2, dtype=torch.float64, device="cuda")
    nb = 2048
    np_ = max(1, (1 << 25) // nb)
    for b in range(0, half.numel(), nb):
        for p in range(0, case["npix"], np_):
            ph = 2 * math.pi * torch.frac(S[p:p + np_] @ U[b:b + nb].T)
            wt = B[p:p + np_, None]
            if case["blockage"]:
                wt = wt * _seen([a[p:p + np_] for a in xyz], t, half[b:b + nb])
            V[b:b + nb, 0] += (wt * torch.cos(ph)).sum(0)
            V[b:b + nb, 1] -= (wt * torch.sin(ph)).sum(0)
    return V.reshape(-1)


def _groups(case, t, V):
    """Groups of every segment as the library forms them: plane fit, grid, keys, stable order, representative."""
    nbl = case["nsat"] * (case["nsat"] - 1) // 2
    u, v, w = (t[k].cpu().numpy() for k in "uvw")
    Vh = V.double().cpu().numpy()
    lam, f32 = np.float32(case["lam"]), np.float32
    bl_max = f32(_bl_max(case, t))
    for t0, tl in zip(*_segments(case)):
        full = np.arange(2 * nbl * t0, 2 * nbl * (t0 + tl))
        q = [a[full].astype(np.longdouble) for a in (u, v, w)]
        uu, vv, uv, uw, vw = ((a * b).sum() for a, b in ((q[0], q[0]), (q[1], q[1]), (q[0], q[1]), (q[0], q[2]), (q[1], q[2])))
        den = uu * vv - uv * uv
        if abs(den) < 1e-24 * uu * vv:
            den = (1 if den >= 0 else -1) * 1e-24 * uu * vv
        fa, fb = f32((vv * uw - uv * vw) / den), f32((uu * vw - uv * uw) / den)
        span = f32(f32(2) * bl_max) / lam
        if case["grid_res"]:
            res = case["grid_res"] | 1
        else:
            r = np.ceil(f32(span * f32(2)) * max(np.sqrt(f32(1) + fa * fa), np.sqrt(f32(1) + fb * fb)))
            res = int(r + 3 - np.fmod(r, f32(2)))
        du = f32(span / f32(res - 1))
        inv = f32(1) / du
        h = (res - 1) // 2
        idx = np.concatenate([np.arange(s * 2 * nbl, s * 2 * nbl + nbl) for s in range(t0, t0 + tl)]) if case["mirror"] else full
        cell = []
        for a in (u, v):
            x = a[idx].astype(np.float64) * np.float64(inv)
            if case["mirror"]:
                c = np.floor((x + 0.5).astype(f32))
            else:
                c = np.where(x >= 0, np.floor((x + 0.5).astype(f32)), np.ceil((x - 0.5).astype(f32)))
            cell.append(c.astype(np.int64) + h)
        inside = (cell[0] >= 0) & (cell[0] < res) & (cell[1] >= 0) & (cell[1] < res)
        key = np.where(inside, cell[0] * res + cell[1] + 1, 0)
        order = np.argsort(key, kind="stable")
        starts = np.flatnonzero(np.r_[True, np.diff(key[order]) != 0])
        counts = np.diff(np.r_[starts, key.size])
        gkey = key[order][starts]
        k0 = gkey - 1
        ugu, vgu = ((k0 // res - h).astype(f32) * du), ((k0 % res - h).astype(f32) * du)
        step, j = idx // (2 * nbl), idx % (2 * nbl)
        val = Vh[step * nbl + j % nbl].copy()
        val[j >= nbl, 1] *= -1
        if case["blockage"]:
            rep = order[starts + counts // 2]
            yield fa, fb, gkey, ugu, vgu, val[rep], idx[rep]
        else:
            mean = np.add.reduceat(val[order], starts, axis=0) / counts[:, None]
            yield fa, fb, gkey, ugu, vgu, mean.astype(f32).astype(np.float64), None


def _exact_image(case, seed):
    xyz = [a.float() for a in _nest_xyz(case["nside"], case["base"], case["npix"])]
    t = _baselines(case, seed)
    l, m, n = (a.double() for a in xyz)
    acc = torch.zeros(case["npix"], dtype=torch.float64, device="cuda")
    W = torch.zeros(case["npix"], dtype=torch.int64, device="cuda")
    total = 0
    for fa, fb, key, ugu, vgu, val, rep in _groups(case, t, _visibilities(case, t, seed)):
        total += key.size
        keep = np.flatnonzero(key != 0)
        for g in np.array_split(keep, max(1, keep.size // 1024)):
            if not g.size:
                continue
            a, b = (torch.from_numpy(x[g].astype(np.float64)).cuda() for x in (ugu, vgu))
            re, im = (torch.from_numpy(val[g, k].copy()).cuda() for k in (0, 1))
            at = torch.from_numpy(rep[g]).cuda() if rep is not None else None
            for p in range(0, case["npix"], 1 << 15):
                sl = slice(p, p + (1 << 15))
                ph = 2 * math.pi * torch.frac((l[sl] + float(fa) * n[sl])[:, None] * a + (m[sl] + float(fb) * n[sl])[:, None] * b)
                term = re * torch.cos(ph) - im * torch.sin(ph)
                if at is not None:
                    ok = _seen([c[sl] for c in xyz], t, at)
                    term = term * ok
                    W[sl] += ok.sum(1)
                acc[sl] += term.sum(1)
    if case["blockage"]:
        image = torch.where(W > 0, acc / W.clamp(min=1), torch.zeros_like(acc))
        return {"C": image, "W": W.to(torch.int32)}
    return {"C": acc / max(1, total), "W": None}
