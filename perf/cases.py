"""Performance cases: the work a user has this framework do, over its range.

Every case goes through the public entry points (the Python mirror
``psod_b200.sod`` and the C-ABI of ``include/psod.h`` through
``psod_b200.capi``) on seeded NFW-mixture boxes of ``psod_b200.synth`` (halo
sizes N^-1.9, 45 % of the particles in halos), which is what the path meets.
Kinds:

  static   psod_cic_rho_static: density of a small zone, no allocation
  density  load + cic + cicm1 + tri_cic: densities and the seed order
  sod      load + cic + cicm1 + tri_cic + spherover + the halo table
  fof      load + psod_fof + the catalogue
  props    haloanalyzer's properties of every halo of a FoF catalogue
  learn    the bracket network's forward and gradient on a batch of samples

``buffers`` "host" is a program whose particles and results are numpy arrays;
"device" one that keeps them on the GPU (device pointers in the C-ABI).
"""

import ctypes as C
import math

import numpy as np
import torch

from psod_b200 import capi, synth
from psod_b200.sod import HaloTable, SphericalOverdensity, _ptr

MODES = {"plain": capi.MODE_PLAIN, "batched": capi.MODE_BATCHED, "learned": capi.MODE_LEARNED}
MPC = 3.08568e24
UNITS = dict(unit_l=MPC * 100 / 0.7, unit_d=2.7e-30, unit_t=4.4e17, aexp=1.0, h0=70.0, hz=1.0, delta_vir=178.0)


def listed():
    return [
        # the smallest call: one rank's 64^3 zone, density only, where launches and latency count
        dict(name="static_64", kind="static", nx=64, nmax=2000),
        # densities and seeds of a mid-sized box, grid a power of two (RAMSES levels)
        dict(name="density_256", kind="density", nx=256, nmax=20000),
        # the same on a grid that is neither a power of two nor a multiple of the tile
        dict(name="density_150", kind="density", nx=150, nmax=20000),
        # a test-sized box with the default parameters (plain mode), results on the host
        dict(name="sod_48_default", kind="sod", nx=48, nmax=6000, nmin=20, mode="plain", buffers="host"),
        # the 128^3 configuration (Mmin 100, Delta 200, 32 bins) of a host program
        dict(name="sod_128_host", kind="sod", nx=128, nmax=20000, nmin=100, mode="batched", nbins=32, rbin_hi=2.0,
             buffers="host"),
        # the default (plain) mode on a larger box, 60 bins
        dict(name="sod_256_plain", kind="sod", nx=256, nmax=20000, nmin=100, mode="plain", buffers="device"),
        # the 512^3 configuration: -npu 2e5, three thresholds in one pass, 48 bins, learned bracket
        dict(name="sod_512_learned", kind="sod", nx=512, nmax=200000, npu=200000, nmin=100, mode="learned", nbins=48,
             deltas=3, buffers="device"),
        # heavy tail: clusters of 5e5 particles, Delta 200/500, 64 bins
        dict(name="sod_256_heavy", kind="sod", nx=256, nmax=50000, npu=1000000, nmin=100, mode="batched", nbins=64,
             deltas=2, clusters=4, cluster_size=500000, buffers="device"),
        # one of the 4^3 zones of the 512^3 box with its buffer: a rank of the zone decomposition
        dict(name="zone_512_4", kind="sod", nx=512, nmax=200000, npu=200000, nmin=100, mode="batched", nbins=48,
             deltas=3, nxcpu=4, nzone=21, buffers="device"),
        # the halo finder with its usual linking length and smallest halo
        dict(name="fof_256", kind="fof", nx=256, nmax=50000, b=0.2, mmin=20),
        # halo properties of a catalogue
        dict(name="props_192", kind="props", nx=192, nmax=50000, b=0.2, mmin=100),
        # one full set of bracket samples through the network, forward and backward
        dict(name="learn_20k", kind="learn", n=20011),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A box side: a power of two, a multiple of eight or any number."""
    nx = _log_int(rng, lo, hi)
    how = rng.randrange(3)
    if how == 0:
        nx = 1 << round(math.log2(nx))
    elif how == 1:
        nx = 8 * round(nx / 8)
    return min(max(nx, lo), hi)


def draw(rng):
    kind = rng.choice(["static", "density", "sod", "sod", "host", "zone", "heavy", "fof", "props", "learn"])
    if kind == "static":
        return dict(kind="static", nx=rng.randint(9, 63), nmax=_log_int(rng, 300, 2000))
    if kind == "learn":
        return dict(kind="learn", n=_log_int(rng, 300, 80000))
    if kind == "fof":
        return dict(kind="fof", nx=_grid(rng, 48, 288), nmax=_log_int(rng, 2000, 50000),
                    b=rng.choice([0.15, 0.2, 0.25]), mmin=rng.choice([10, 20, 100]))
    if kind == "props":
        return dict(kind="props", nx=_grid(rng, 48, 192), nmax=_log_int(rng, 2000, 50000), b=0.2,
                    mmin=rng.choice([50, 100]))
    if kind == "density":
        return dict(kind="density", nx=_grid(rng, 24, 320), nmax=_log_int(rng, 2000, 20000))
    nmin = rng.choice([20, 50, 100])
    if kind == "host":
        return dict(kind="sod", nx=_grid(rng, 32, 144), nmax=_log_int(rng, 2000, 15000), nmin=nmin,
                    mode=rng.choice(["plain", "batched"]), nbins=rng.choice([32, 60]), buffers="host")
    if kind == "zone":
        k = rng.choice([3, 4])
        return dict(kind="sod", nx=k * 8 * rng.randint(5, 10), nmax=_log_int(rng, 2000, 15000), nmin=nmin,
                    mode="batched", nbins=48, deltas=rng.choice([1, 3]), nxcpu=k, nzone=rng.randrange(k**3),
                    buffers="device")
    if kind == "heavy":
        size = _log_int(rng, 100000, 400000)
        return dict(kind="sod", nx=8 * rng.randint(20, 30), nmax=20000, npu=2 * size, nmin=100, mode="batched",
                    nbins=64, deltas=2, clusters=rng.choice([1, 2, 3]), cluster_size=size, buffers="device")
    mode = rng.choice(["plain", "batched", "learned"])
    npu = _log_int(rng, 20000, 200000)
    return dict(kind="sod", nx=_grid(rng, 48, 224 if mode == "plain" else 352), nmax=int(0.6 * npu), npu=npu,
                nmin=nmin, mode=mode, nbins=rng.choice([32, 48, 60]), deltas=rng.choice([1, 2, 3]), buffers="device")


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _box(case, seed):
    clusters = dict(n_clusters=case["clusters"], cluster_size=case["cluster_size"]) if case.get("clusters") else {}
    box = synth.make_box(case["nx"], nmax_halo=case["nmax"], seed=seed, device="cuda", **clusters)
    pos, ids = box.pos, box.ids
    del box
    torch.cuda.empty_cache()  # the generator's temporaries: the engine allocates its own memory
    return pos, ids


def _vel(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    return 0.3 * torch.randn(n, 3, generator=g, device="cuda")


def _zone_buffer(case):
    """Buffer cells of a zone context: from -npu, else half a zone."""
    if case.get("npu"):
        return 4 * math.ceil((case["npu"] * 2.0 / 200.0) ** (1 / 3) / 2.0)
    return case["nx"] // case["nxcpu"] // 2


def _zone_side(case):
    return min(case["nx"], case["nx"] // case["nxcpu"] + 2 * _zone_buffer(case))


def _select_zone(pos, ids, nx, k, nzone, nxb):
    """The particles of one zone and its buffer (the FP64 test of psod_select_zone)."""
    nxzone = nx // k
    rs = (0.5 + nxb / nxzone) / k
    keep = torch.ones(pos.shape[0], dtype=torch.bool, device=pos.device)
    for a, i in enumerate((nzone // (k * k), (nzone // k) % k, nzone % k)):
        d = (pos[:, a].double() - ((i / k) + ((i + 1) / k)) / 2.0).abs()
        keep &= (d < rs) | (d > 1.0 - rs)
    return pos[keep].contiguous(), ids[keep].contiguous()


def _bracket(params):
    """A bracket model trained on the samples of one 96^3 box."""
    box = synth.make_box(96, nmax_halo=20000, seed=7, device="cuda")
    own = dict(params, mode=capi.MODE_BATCHED, npu=0)
    with SphericalOverdensity(96, **own) as s:
        s.learn_collect(1 << 18)
        s.load(box.pos, box.ids)
        s.run()
        s.learn_train(epochs=10, batch=256, lr=1e-3, seed=1)
        return s.learn_get_model()


# Result arrays are made once, as large as the box can need (what a program does that cannot know the halo count before
# the call), and zero beyond what a pass writes.
def _halo_buffers(n, nmin, nbins, ndelta, host):
    h, m = n // (2 * nmin) + 64, 3 * n // 5 + 64

    def new(k, dt="int64"):
        return np.zeros(max(1, k), dt) if host else torch.zeros(max(1, k), dtype=getattr(torch, dt), device="cuda")

    return HaloTable(halo_id=new(h), halo_mass=new(h), halo_rank=new(h), halo_center=new(3 * h, "float32"),
                     halo_rdelta=new(h, "float64"), halo_mass2=new(h), halo_mextra=new(h * ndelta),
                     halo_profile=new(h * nbins), member_offset=new(h + 1), member_index=new(m), member_id=new(m))


def _model(seed):
    """A random bracket model in the blob's layout (psod.h): scales, then padded weights and biases."""
    r = np.random.default_rng(seed)
    w1, w2, w3 = np.zeros((64, 16)), r.normal(0, 0.18, (64, 64)), np.zeros((8, 64))
    w1[:, :10] = r.normal(0, 0.45, (64, 10))
    w3[:2] = r.normal(0, 0.1, (2, 64))
    b1, b2, b3 = r.normal(0, 0.1, 64), r.normal(0, 0.1, 64), np.zeros(8)
    mu, sg, my, sy = np.zeros(16), np.ones(16), r.normal(0, 0.5, 2), np.array([0.6, 1.2])
    mu[:10], sg[:10] = r.normal(0, 1.0, 10), 0.5 + r.random(10)
    return np.concatenate([a.ravel() for a in (mu, sg, my, sy, w1, b1, w2, b2, w3, b3)]).astype(np.float32)


def _learn_inputs(case, seed):
    r = np.random.default_rng(seed)
    blob = _model(seed)
    x = (blob[:10] + blob[16:26] * r.normal(0, 1, (case["n"], 10))).astype(np.float32)
    t = (blob[32:34] + blob[34:36] * r.normal(0, 1, (case["n"], 2))).astype(np.float32)
    return blob, x, t


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "learn":
        s["blob"], s["x"], s["t"] = _learn_inputs(case, seed)
        s["so"] = SphericalOverdensity(32, mode=capi.MODE_LEARNED)
        s["so"].learn_set_model(s["blob"])
        return s
    pos, ids = _box(case, seed)
    n = pos.shape[0]
    if kind == "static":
        s.update(lib=capi.load(), pos=pos, rho=torch.empty(n, dtype=torch.float64, device="cuda"))
        return s
    if kind == "sod":
        ndelta = case.get("deltas", 1) - 1
        params = dict(nmin=case["nmin"], mode=MODES[case["mode"]], nbins=case.get("nbins", 60),
                      npu=case.get("npu", 0), rbin_hi=case.get("rbin_hi", 1.0), delta_extra=(500.0, 178.0)[:ndelta])
        k = case.get("nxcpu", 1)
        s["total"] = n
        if k > 1:
            pos, ids = _select_zone(pos, ids, case["nx"], k, case["nzone"], _zone_buffer(case))
            torch.cuda.empty_cache()
            n = 3 * _zone_side(case) ** 3 // 2
            params.update(nxcpu=k, nzone=case["nzone"])
        model = _bracket(dict(params)) if case["mode"] == "learned" else None
        s["so"] = SphericalOverdensity(case["nx"], **params)
        if model is not None:
            s["so"].learn_set_model(model)
        host = case["buffers"] == "host"
        s.update(pos=pos.cpu().numpy() if host else pos, ids=ids.cpu().numpy() if host else ids,
                 out=_halo_buffers(n, case["nmin"], params["nbins"], ndelta, host))
        return s
    s.update(so=SphericalOverdensity(case["nx"]), pos=pos, ids=ids)
    if kind == "density":
        s.update(rho=torch.empty(n, dtype=torch.float64, device="cuda"),
                 isort=torch.zeros(n, dtype=torch.int64, device="cuda"))
        return s
    s["vel"] = _vel(n, seed)
    if kind == "fof":
        h = n // case["mmin"] + 1
        i64 = lambda k: torch.zeros(k, dtype=torch.int64, device="cuda")  # noqa: E731
        f64 = lambda *k: torch.zeros(*k, dtype=torch.float64, device="cuda")  # noqa: E731
        s["out"] = dict(halo_id=i64(h), halo_mass=i64(h), halo_com=f64(h, 3), halo_vel=f64(h, 3), halo_radius=f64(h),
                        member_offset=i64(h + 1), member_index=i64(n), member_id=i64(n))
        return s
    so = s["so"]
    so.load(pos, ids, vel=s["vel"])
    nh = so.fof(percolation=case["b"], mmin=case["mmin"])["nhalo"]
    p = capi.PropsParams(*(UNITS[f] for f in ("unit_l", "unit_d", "unit_t", "aexp", "h0", "hz", "delta_vir")),
                         _levelmin(case), 0, 1, capi.PROPS_FROM_FOF, 30000, 0)
    cap = _props_rows(case)
    if nh > cap:
        raise RuntimeError(f"{nh} halos, room for {cap}")
    s.update(params=p, out={f: torch.zeros((cap, k) if k > 1 else cap, dtype=getattr(torch, dt), device="cuda")
                            for f, k, dt in capi.PROPS_FIELDS})
    return s


def _props_rows(case):
    return case["nx"] ** 3 // (4 * case["mmin"]) + 64


def _levelmin(case):
    return round(math.log2(case["nx"]))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ok(st):
    if st != capi.OK:
        raise RuntimeError(f"psod status {st}")


def _table(cls, out):
    t = cls()
    for f, a in out.items():
        setattr(t, f, a.data_ptr())
    return t


def run(s):
    kind = s["kind"]
    if kind == "static":
        _ok(s["lib"].psod_cic_rho_static(s["pos"].shape[0], _ptr(s["pos"]), s["case"]["nx"], 0, 0, _ptr(s["rho"]), None,
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s["rho"]
    so = s["so"]
    if kind == "learn":
        grad, loss = so.learn_gradient(s["x"], s["t"])
        return dict(y=so.learn_forward(s["x"]), grad=grad, loss=loss)
    if kind == "props":
        _ok(so.lib.psod_halo_properties(so.ctx, C.byref(s["params"]), None))
        t = _table(capi.PropsTable, s["out"])
        _ok(so.lib.psod_props_get(so.ctx, C.byref(t)))
        return s["out"]
    if kind == "fof":
        so.load(s["pos"], s["ids"], vel=s["vel"])
        so.fof(percolation=s["case"]["b"], mmin=s["case"]["mmin"])
        t = _table(capi.FofTable, s["out"])
        _ok(so.lib.psod_fof_get_halos(so.ctx, C.byref(t)))
        return s["out"]
    if kind == "density":
        so.load(s["pos"], s["ids"])
        so.cic()
        _ok(so.lib.psod_cicm1(so.ctx, _ptr(s["rho"])))
        nn = C.c_int64(0)
        _ok(so.lib.psod_tri_cic(so.ctx, _ptr(s["isort"]), C.byref(nn)))
        return dict(rho=s["rho"], isort=s["isort"])
    so.load(s["pos"], s["ids"], npart_total=s["total"])
    so.run()
    so.halos(out=s["out"])
    return vars(s["out"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _power_moment(nmin, nmax, p):
    """Mean of N^p under dN/dN_h ~ N^-1.9 on [nmin, nmax]."""
    a, b = p - 0.9, -0.9
    return ((nmax**a - nmin**a) / a) / ((nmax**b - nmin**b) / b)


def work(case):
    kind = case["kind"]
    if kind == "learn":  # three layers forward, twice that backward, forward again; samples in, outputs out
        n = case["n"]
        return dict(bytes=n * 4 * (10 + 2 + 2) + 4 * 5768, flops=n * 2 * 5760 * 4)
    n = case["nx"] ** 3
    if kind == "static":  # 12 B in, 8 B out; 8 weights of 2 products, deposited and gathered
        return dict(bytes=20 * n, flops=n * 8 * 6)
    if kind == "density":  # positions in, densities out, half the particles as seeds
        return dict(bytes=n * (12 + 8 + 8 + 4), flops=n * 8 * 6)
    if kind == "fof":  # positions, IDs and velocities in; members (about 40 %) out
        return dict(bytes=n * (12 + 8 + 12 + 0.4 * 16), flops=n * 60)
    # pairs of the halos' members, from the halo law
    halo = 0.45 * n
    if kind == "props":  # potential: every ordered pair of a halo, 3 differences, 3 squares, softening, root, quotient
        top = min(case["nmax"], 30000)
        pairs = halo * _power_moment(20, top, 2) / _power_moment(20, case["nmax"], 1)
        return dict(bytes=halo * (12 + 12 + 4), flops=10 * pairs)
    if case.get("nxcpu", 1) > 1:
        n = _zone_side(case) ** 3
    # particles in, members and the table out; the members' distances to their centre
    return dict(bytes=n * (12 + 8) + 0.3 * n * 16, flops=0.3 * n * 10)


# ---------------------------------------------------------------------------
# the values in 64 bits
# ---------------------------------------------------------------------------
def _rho64(pos, nx):
    """CIC density on the (2 nx)^3 periodic nodes, interpolated back."""
    nc, n = 2 * nx, pos.shape[0]
    g = pos.double() * nc
    i0 = torch.floor(g)
    d = g - i0
    lo = i0.long() % nc
    hi = (lo + 1) % nc
    del g, i0
    grid = torch.zeros(nc**3, dtype=torch.float64, device=pos.device)

    def corners():
        for c in range(8):
            ax = [(hi[:, a], d[:, a]) if (c >> a) & 1 else (lo[:, a], 1.0 - d[:, a]) for a in range(3)]
            yield ax[0][0] + nc * (ax[1][0] + nc * ax[2][0]), ax[0][1] * ax[1][1] * ax[2][1]

    for node, w in corners():
        grid.index_add_(0, node, w)
    rho = torch.zeros(n, dtype=torch.float64, device=pos.device)
    for node, w in corners():
        rho += grid[node] * w
    return rho * (float(nc) ** 3 / n)


def _components(lab, a, b):
    """Joins the components of the edges (a, b) in the labels (every label a root)."""
    while a.numel():
        la, lb = lab[a], lab[b]
        on = la != lb
        a, b, la, lb = a[on], b[on], la[on], lb[on]
        lo, hi = torch.minimum(la, lb), torch.maximum(la, lb)
        lab.scatter_reduce_(0, hi, lo, "amin")
        while True:
            up = lab[lab]
            if torch.equal(up, lab):
                break
            lab.copy_(up)


def _groups(pos, b, nres):
    """Group label of every particle: friends are pairs with a minimum-image FP32 distance <= b/nres.  Cells with a
    diagonal below that length are single nodes; neighbouring cells are joined by their particle pairs."""
    rT = np.float32(b) / np.float32(nres)
    r2 = float(np.float32(rT * rT))
    m = int(math.ceil(math.sqrt(3.0) / (float(rT) * (1 - 1e-4)))) + 1
    pos = torch.where(pos == 1.0, torch.zeros_like(pos), pos)
    ci = (pos.double() * m).long().clamp_(0, m - 1)
    key, order = torch.sort(ci[:, 0] + m * (ci[:, 1] + m * ci[:, 2]))
    p = pos[order]
    del ci
    cell, cnt = torch.unique_consecutive(key, return_counts=True)
    start = torch.cumsum(cnt, 0) - cnt
    node = torch.repeat_interleave(torch.arange(cell.numel(), device=pos.device), cnt)
    lab = torch.arange(cell.numel(), device=pos.device)
    cx, cy, cz = cell % m, (cell // m) % m, cell // (m * m)

    def friends(i, j):
        d = (p[i] - p[j]).abs()
        d = torch.where(d > 0.5, 1.0 - d, d)
        q = d * d
        return (q[:, 0] + q[:, 1]) + q[:, 2] <= r2

    def join(u, v, most):
        """Tests up to `most` x `most` particle pairs of each pair of cells; returns the pairs of cells not joined."""
        for s in range(0, u.numel(), 1 << 20):
            a, c = u[s:s + (1 << 20)], v[s:s + (1 << 20)]
            na, nc = cnt[a].clamp(max=most), cnt[c].clamp(max=most)
            tot = torch.cumsum(na * nc, 0)
            at = 0
            while at < a.numel():
                base = int(tot[at - 1]) if at else 0
                to = max(at + 1, int(torch.searchsorted(tot, torch.tensor(base + (1 << 26), device=tot.device))))
                aa, cc = a[at:to], c[at:to]
                w = torch.repeat_interleave(torch.arange(aa.numel(), device=aa.device), na[at:to] * nc[at:to])
                k = torch.arange(w.numel(), device=w.device) - (tot[at:to] - na[at:to] * nc[at:to] - base)[w]
                hit = friends(start[aa[w]] + k // nc[at:to][w], start[cc[w]] + k % nc[at:to][w])
                got = torch.unique(w[hit])
                _components(lab, aa[got], cc[got])
                at = to
        on = lab[u] != lab[v]
        return u[on], v[on]

    for most in (2, 1 << 30):  # a few pairs first: they join most of every large group
        for oz in range(0, 3):
            for oy in range(-2 if oz else 0, 3):
                for ox in range(-2 if oz or oy else 1, 3):
                    want = (cx + ox) % m + m * ((cy + oy) % m + m * ((cz + oz) % m))
                    at = torch.searchsorted(cell, want).clamp_(max=cell.numel() - 1)
                    u = torch.nonzero((cell[at] == want) & (lab != lab[at])).squeeze(1)
                    join(u, at[u], most)
    out = torch.empty(pos.shape[0], dtype=torch.int64, device=pos.device)
    out[order] = lab[node]
    return out


def _catalogue(pos, ids, b, nres, mmin):
    """(members in catalogue order, halo of each, masses) of the groups of at least mmin particles."""
    lab = _groups(pos, b, nres)
    n = pos.shape[0]
    size = torch.bincount(lab, minlength=n)
    low = torch.full((n,), n, dtype=torch.int64, device=pos.device)
    low.scatter_reduce_(0, lab, torch.arange(n, device=pos.device), "amin")
    root = torch.nonzero(size >= mmin).squeeze(1)
    root = root[torch.argsort(ids[low[root]])]
    rank = torch.full((n,), -1, dtype=torch.int64, device=pos.device)
    rank[root] = torch.arange(root.numel(), device=pos.device)
    halo = rank[lab]
    mem = torch.nonzero(halo >= 0).squeeze(1)
    halo, by = torch.sort(halo[mem], stable=True)
    return mem[by], halo, size[root]


def _rows(v, rows):
    """Zero rows beyond the halos, as in the result arrays."""
    return torch.cat([v, v.new_zeros((rows - v.shape[0],) + v.shape[1:])])


def _sum(v, halo, nh):
    return torch.zeros((nh,) + v.shape[1:], dtype=torch.float64, device=v.device).index_add_(0, halo, v)


def _max(v, halo, nh):
    return torch.zeros(nh, dtype=torch.float64, device=v.device).scatter_reduce_(0, halo, v, "amax")


def _exact_fof(case, seed):
    pos, ids = _box(case, seed)
    vel = _vel(pos.shape[0], seed)
    mem, halo, mass = _catalogue(pos, ids, case["b"], case["nx"], case["mmin"])
    nh = mass.numel()
    x, first = pos[mem].double(), torch.cumsum(mass, 0) - mass
    dl = x[first][halo] - x
    com = _sum(x + (dl > 0.5).double() - (dl < -0.5).double(), halo, nh) / mass[:, None]
    com = com - (com > 1.0).double() + (com < 0.0).double()
    d = (x - com[halo]).abs()
    d = torch.where(d > 0.5, 1.0 - d, d)
    rows = pos.shape[0] // case["mmin"] + 1
    return dict(halo_id=None, halo_mass=None, halo_com=_rows(com, rows),
                halo_vel=_rows(_sum(vel[mem].double(), halo, nh) / mass[:, None], rows),
                halo_radius=_rows(_max((d * d).sum(1), halo, nh).sqrt(), rows), member_offset=None, member_index=None,
                member_id=None)


def _potential(x, mass, first, eps2):
    """Sum over a halo's members of the other members' 1/sqrt(d^2 + eps2)."""
    out = torch.zeros(mass.numel(), dtype=torch.float64, device=x.device)
    for h, (k, b) in enumerate(zip(mass.tolist(), first.tolist())):
        if k >= 30000:  # the sampled potential of large halos
            at = b + (torch.arange(3000, device=x.device) * k) // 3000
            k, y = 3000, x[at]
        else:
            y = x[b:b + k]
        for i in range(0, k, 4096):
            q = y[i:i + 4096]
            d2 = sum((q[:, None, a] - y[None, :, a]) ** 2 for a in range(3))
            out[h] += torch.rsqrt(d2 + eps2).sum()
        out[h] -= k / math.sqrt(eps2)  # a member with itself
    return out


def _exact_props(case, seed):
    pos, ids = _box(case, seed)
    vel = _vel(pos.shape[0], seed)
    mem, halo, mass = _catalogue(pos, ids, case["b"], case["nx"], case["mmin"])
    nh, np_ = mass.numel(), mass.double()
    u, lev = UNITS, _levelmin(case)
    mp, G, pi = 2.0 ** (-3 * lev), float(np.float32(6.6731e-08)), float(np.float32(3.14159265359879))
    f43, third = float(np.float32(4.0 / 3.0)), float(np.float32(1.0 / 3.0))
    msun, first = 1.98892e33, torch.cumsum(mass, 0) - mass
    # periodic unwrap: halos over more than half the box keep their upper part one box down
    x32 = pos[mem].clone()
    for a in range(3):
        c = x32[:, a]
        hi = torch.full((nh,), -1.0, device=c.device).scatter_reduce_(0, halo, c, "amax")
        lo = torch.full((nh,), 2.0, device=c.device).scatter_reduce_(0, halo, c, "amin")
        x32[:, a] = torch.where(((hi - lo) > 0.5)[halo] & (c > 0.5), c - 1.0, c)
    com = _sum(x32.double(), halo, nh) / np_[:, None]
    below = com < 0.0
    com = com + below.double()
    x32 = torch.where(below[halo], x32 + 1.0, x32)
    x = x32.double()
    comv = _sum(vel[mem].double(), halo, nh) / np_[:, None]
    q, v = x - com[halo], vel[mem].double() - comv[halo]
    r2 = (q * q).sum(1)
    w2 = ((v + u["hz"] * q) ** 2).sum(1)
    m_vir = np_ * mp * u["unit_d"] * u["unit_l"] ** 3
    r_vir = (3 * m_vir / (4 * pi * u["delta_vir"] * u["unit_d"])) ** third
    v_vir = (G * m_vir / r_vir).sqrt()
    vu = u["unit_l"] / u["unit_t"]
    dispv2 = _sum(w2, halo, nh)
    ekin = 0.5 * mp * dispv2 * u["unit_d"] * u["unit_l"] ** 5 / u["unit_t"] ** 2
    eps = float(np.float32(np.float32(1.0 / 2.0**lev) * np.float32(1.0 / 64.0)))
    pot = mp * mp * _potential(x, mass, first, eps * eps)
    many = torch.where(mass < 30000, torch.ones_like(np_), (np_ * np_ - np_) / (3000.0 * 3000.0 - 3000.0))
    epot = -0.5 * G * pot * (u["unit_d"] * u["unit_l"] ** 3) ** 2 / u["unit_l"] * many
    ev = 0.5 * m_vir / msun * (v_vir / 1e5) ** 2
    ang = _sum(mp * torch.linalg.cross(q, v), halo, nh) * u["unit_d"] * u["unit_l"] ** 5 / u["unit_t"]
    inertia = _sum(q[:, :, None] * q[:, None, :], halo, nh) / np_[:, None, None]
    eig = torch.linalg.eigvalsh(inertia).flip(1).clamp(min=0).sqrt()
    out = dict.fromkeys(f for f, _, _ in capi.PROPS_FIELDS)
    h = u["h0"] / 100.0
    out.update(
        mvir=m_vir / msun * h, rvir=r_vir / (MPC / 1e3) * h, rvircom=r_vir / (MPC / 1e3) * h / u["aexp"],
        vvir=v_vir / 1e5, com=com * u["unit_l"] / MPC * h / u["aexp"], comv=comv * vu / 1e5,
        rmax=_max(r2, halo, nh).sqrt() * u["unit_l"] / r_vir, vmax=_max(w2, halo, nh).sqrt() * vu / v_vir,
        dispx=(_sum(r2, halo, nh) / np_).sqrt() * u["unit_l"] / r_vir, dispv=(dispv2 / np_).sqrt() * vu / v_vir,
        ekin=ekin / (msun * 1e10) / ev, epot=epot / (msun * 1e10) / ev, eig_val=eig * u["unit_l"] / r_vir[:, None])
    out["lambda"] = ang * (ekin + epot).abs().sqrt()[:, None] / (G * m_vir**2.5)[:, None]
    out["lambda_prime"] = ang / (float(np.float32(math.sqrt(2.0))) * m_vir * r_vir * v_vir)[:, None]
    return {f: None if a is None else _rows(a, _props_rows(case)) for f, a in out.items()}


def _exact_learn(case, seed):
    blob, x, t = (torch.from_numpy(a).double() for a in _learn_inputs(case, seed))
    xs, ts = (x - blob[:10]) / blob[16:26], (t - blob[32:34]) / blob[34:36]
    sizes = [(64, 16), (64,), (64, 64), (64,), (8, 64), (8,)]
    par = [p.clone().reshape(s).requires_grad_() for p, s in zip(blob[36:].split([math.prod(s) for s in sizes]), sizes)]
    w1, b1, w2, b2, w3, b3 = par
    y = torch.relu(torch.relu(xs @ w1[:, :10].T + b1) @ w2.T + b2) @ w3[:2].T + b3[:2]
    loss = 0.5 * ((y - ts) ** 2).sum() / case["n"]
    loss.backward()
    return dict(y=(y.detach() * blob[34:36] + blob[32:34]), grad=torch.cat([p.grad.flatten() for p in par]),
                loss=float(loss.detach()))


def exact(case, seed):
    """What run() returns, in 64 bits with plain torch.  The SOD table has none: its floating values are a chosen
    particle's position and distance, which follow from whole-number decisions over the box."""
    kind = case["kind"]
    if kind == "static":
        return _rho64(_box(case, seed)[0], case["nx"])
    if kind == "density":
        return dict(rho=_rho64(_box(case, seed)[0], case["nx"]), isort=None)
    if kind == "fof":
        return _exact_fof(case, seed)
    if kind == "props":
        return _exact_props(case, seed)
    if kind == "learn":
        return _exact_learn(case, seed)
    return None
