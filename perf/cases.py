"""The framework's work as its users call it: light rays through a cone octree
(the hmaps, catalogues and rays drivers), the octree's creation from cells
(create_octree) and the velocity-field deposit.

Inputs are seeded synthetic cones of the benchmark's construction, made on the
GPU: a periodic Gaussian random field over a 2048 Mpc/h box, refined in NFW
haloes, 48-byte records sorted by key, flat LCDM.  A case's haloes, and so its
cells, stay where they are; another seed is another field in them and other
ray directions, sources, particles or cell file order.
"""
from __future__ import annotations

import ctypes as C
import importlib
import math

import numpy as np
import torch

PKG = "magrathea-pathfinder_gb300"
CLIGHT, MPC, GN, MSUN = 299792458.0, 3.08568e22, 6.674e-11, 1.98847e30
HUB, OM, LBOX = 0.68, 0.31, 2048.0
H0 = HUB * 1e5 / MPC
LENGTH = LBOX * MPC / HUB
HALF = 5.0                      # the cone's half opening, degrees
DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an interactive call or a test: a handful of rays through a small uniform cone, CIC, no lensing
        dict(name="rays_few", kind="rays", n=64, base=8, top=8, halos=0, z=0.2, nsteps=10, order=1, planes=0, jac=False,
             exact=False, vel=False, device=False),
        # the uniform 64^3 field with 4096 rays to z = 0.5, CIC: the smallest of the standard workloads
        dict(name="rays_cone_cic", kind="rays", n=4096, base=8, top=8, halos=0, z=0.5, nsteps=10, order=1, planes=0,
             jac=False, exact=False, vel=False, device=False),
        # an ordinary tomographic call on an AMR cone: an odd number of rays, TSC, three surfaces with lensing, host arrays
        dict(name="rays_amr_tsc", kind="rays", n=20011, base=9, top=12, halos=120, z=1.0, nsteps=8, order=2, planes=3,
             jac=True, exact=False, vel=False, device=False),
        # the large survey field: a 400 x 400 grid to z = 2 with the Jacobian, device buffers, the deepest refinement
        dict(name="rays_amr_large", kind="rays", n=160000, base=9, top=13, halos=250, z=2.0, nsteps=8, order=2, planes=1,
             jac=True, exact=False, vel=False, device=True),
        # the nearby velocity-field cone: Doppler redshifts with an observer velocity, two surfaces
        dict(name="rays_velocity", kind="rays", n=8009, base=8, top=10, halos=20, z=0.12, nsteps=5, order=2, planes=2,
             jac=True, exact=False, vel=True, device=False),
        # reference-exact float64 rays, as a validation run or the accuracy statistic makes them
        dict(name="rays_exact", kind="rays", n=4099, base=8, top=10, halos=20, z=0.1, nsteps=8, order=2, planes=1,
             jac=True, exact=True, vel=False, device=False),
        # convergence maps: RING pixels of an nside 2048 map over an AMR cone, two source redshifts
        dict(name="maps", kind="maps", n=60000, base=9, top=12, halos=120, z=1.0, nsteps=8, order=2, planes=2, nside=2048,
             bundle=False),
        # the same map with the four-ray bundle Jacobian
        dict(name="maps_bundle", kind="maps", n=9001, base=8, top=11, halos=40, z=1.0, nsteps=8, order=2, planes=1,
             nside=2048, bundle=True),
        # a halo catalogue: the source positions' observed angles and redshifts, Newton root-finding to 1e-8
        dict(name="catalogue", kind="catalogue", n=16384, base=9, top=12, halos=120, z=1.0, nsteps=8, order=2),
        # the rays driver: trajectories of central rays with their bundles and angular diameter distances
        dict(name="ray_bundles", kind="bundles", n=96, base=8, top=11, halos=40, z=1.0, nsteps=4, order=2, count=8),
        # creation of a cone octree from simulation cells
        dict(name="cells_build", kind="cells", base=9, top=12, halos=120, z=1.0, order=2, dup=0.1, drop=0.01),
        # one shell of particles deposited on the velocity-field octree, TSC at every level
        dict(name="velocity_deposit", kind="deposit", n=500009, base=9, top=12, halos=120, z=1.0, order=2),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "rays", "maps", "maps", "catalogue", "bundles", "cells", "deposit"])
    base = rng.choice([8, 8, 9])
    top = base + rng.choice([0, 1, 2, 3])
    halos = 0 if top == base else _loguniform(rng, 10, 150)
    z = round(math.exp(rng.uniform(math.log(0.2), math.log(1.5))), 3)
    order = rng.choice([1, 2, 2])
    c = dict(kind=kind, base=base, top=top, halos=halos, z=z, nsteps=rng.choice([4, 5, 8, 10]), order=order)
    if kind == "rays":
        exact = rng.random() < 0.2
        jac = rng.random() < 0.7
        c.update(n=_loguniform(rng, 64, 4096 if exact else 100000), planes=rng.randint(1, 4) if jac else rng.randint(0, 1),
                 jac=jac, exact=exact, vel=(not exact) and rng.random() < 0.2, device=rng.random() < 0.4)
        if exact:
            c.update(base=8, top=min(top, 10), halos=min(halos, 20), z=round(rng.uniform(0.06, 0.12), 3))
            if c["top"] <= 8:
                c.update(top=8, halos=0)
    elif kind == "maps":
        bundle = rng.random() < 0.3
        c.update(n=_loguniform(rng, 500, 8000 if bundle else 60000), planes=rng.randint(1, 3),
                 nside=rng.choice([1024, 2048, 4096]), bundle=bundle)
    elif kind == "catalogue":
        c.update(n=_loguniform(rng, 500, 16384))
    elif kind == "bundles":
        c.update(n=_loguniform(rng, 4, 128), count=rng.randint(4, 12), nsteps=4, base=8, z=round(rng.uniform(1.0, 1.4), 3),
                 top=min(top, 11))
        if c["top"] <= 8:
            c.update(top=8, halos=0)
    elif kind == "cells":
        c.update(dup=round(rng.uniform(0.0, 0.2), 3), drop=round(rng.uniform(0.0, 0.05), 3))
        del c["nsteps"]
    else:
        c.update(n=_loguniform(rng, 5000, 500000))
        del c["nsteps"]
    return c


# ---------------------------------------------------------------------------
# the synthetic cone (float64 on the GPU)
# ---------------------------------------------------------------------------
def _efun(a):
    return np.sqrt(OM / a ** 3 + 1.0 - OM)


_z = np.linspace(0.0, 4.0, 40001)
_ez = 1.0 / np.sqrt(OM * (1 + _z) ** 3 + 1 - OM)
_chi = np.concatenate([[0.0], np.cumsum(0.5 * (_ez[1:] + _ez[:-1]) * np.diff(_z))]) * (CLIGHT / 1e5)   # Mpc/h


def _chi_of_z(z):
    return float(np.interp(z, _z, _chi)) / LBOX


def _cosmology(n=4000, amin=0.05):
    aa = np.linspace(1.0, amin, n)
    hh = H0 * _efun(aa)
    dtda = -1.0 / (aa * aa * hh)
    t = np.concatenate([[0.0], np.cumsum(0.5 * (dtda[1:] + dtda[:-1]) * np.diff(aa))])
    return t, aa, -aa * aa * hh


def _interp(x, xp, fp):
    """Linear interpolation on the device in increasing xp."""
    i = torch.searchsorted(xp, x.contiguous()).clamp(1, xp.numel() - 1)
    return fp[i - 1] + (fp[i] - fp[i - 1]) * (x - xp[i - 1]) / (xp[i] - xp[i - 1])


def _spread_table():
    c = torch.arange(1 << 15, device=DEV, dtype=torch.int64)
    s = torch.zeros_like(c)
    for b in range(15):
        s |= ((c >> b) & 1) << (4 * b)
    return s


def _markers():
    m = [0]
    for k in range(15):
        m.append(m[-1] | (8 << (4 * k)))
    return torch.tensor(m, device=DEV, dtype=torch.int64)


def _keys(level, c, table, marks):
    """High words of the 128-bit keys of cells c[..., 3] at `level` (a number or a tensor, at most 15)."""
    k = table[c[..., 0]] + 2 * table[c[..., 1]] + 4 * table[c[..., 2]]
    if isinstance(level, int):
        return (k + marks[level]) << (64 - 4 * level)
    return (k + marks[level]) << (64 - 4 * level)


class Cone:
    """Sorted cells of one synthetic cone: keys, level, centre and fields, on the device."""

    def __init__(self, case, seed):
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) * 1000003 + 17)
        self.table, self.marks = _spread_table(), _markers()
        base, top, nh = case["base"], case["top"], case["halos"]
        self.base, self.top = base, top
        nbox = 1 << (base - 2)
        k = torch.fft.fftfreq(nbox, device=DEV, dtype=F64) * nbox
        kz = torch.fft.rfftfreq(nbox, device=DEV, dtype=F64) * nbox
        kk = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2)
        kk[0, 0, 0] = 1.0
        amp = kk ** -1.5 * torch.exp(-0.5 * (kk / 16.0) ** 2)
        amp[0, 0, 0] = 0.0
        f = torch.fft.irfftn(torch.fft.rfftn(torch.randn((nbox,) * 3, generator=g, device=DEV, dtype=F64)) * amp, s=(nbox,) * 3)
        grid = f / f.std() * (1e-5 * CLIGHT ** 2)
        dx = LENGTH / nbox
        lap = sum(torch.roll(grid, -1, d) + torch.roll(grid, 1, d) for d in range(3)) - 6 * grid
        field = torch.stack([grid] + [(torch.roll(grid, -1, d) - torch.roll(grid, 1, d)) / (2 * dx) for d in range(3)]
                            + [1.0 + 0.3 * lap / lap.std()], dim=-1).reshape(-1, 5)
        xmax = _chi_of_z(case["z"]) * 1.02
        th = math.tan(math.radians(HALF))
        # base cells of the cone with a margin of three cells
        cell = 4.0 / 2 ** base
        pad = 3 * cell

        def cells(lo, hi):
            return torch.arange(int((lo + 2.0) / cell), int((hi + 2.0) / cell) + 1, device=DEV, dtype=torch.int64)

        w = xmax * th + pad
        c = torch.cartesian_prod(cells(-pad - cell, xmax + pad), cells(-w - cell, w + cell), cells(-w - cell, w + cell))
        x = self._centres(base, c)
        keep = ((x[:, 0] > -pad) & (x[:, 0] < xmax + pad) & (x[:, 1].abs() <= x[:, 0].clamp(min=0) * th + pad)
                & (x[:, 2].abs() <= x[:, 0].clamp(min=0) * th + pad)) | (x.abs().amax(1) <= pad + cell)
        levels = [c[keep]]
        hal = None
        if nh:
            gh = torch.Generator(device=DEV)
            gh.manual_seed(4711)
            u = torch.rand((nh, 4), generator=gh, device=DEV, dtype=F64)
            hx = (xmax * u[:, 0] ** (1 / 3)).clamp(min=0.05 * xmax)
            hc = torch.stack([hx, (2 * u[:, 1] - 1) * hx * th, (2 * u[:, 2] - 1) * hx * th], 1)
            mass = torch.exp(math.log(1e12) + u[:, 3] * math.log(1e3))
            r200 = (3 * mass / (4 * math.pi * 200 * 2.775e11)) ** (1 / 3)
            hal = (hc, r200 / LBOX, r200 / 5.0 / LBOX * LENGTH, GN * mass / HUB * MSUN / (math.log(6.0) - 5.0 / 6.0))
            for L in range(base, top):
                x = self._centres(L, levels[-1])
                rad = hal[1] + 4.5 * 4.0 / 2 ** L
                m = torch.zeros(x.shape[0], dtype=torch.bool, device=DEV)
                for h0 in range(0, nh, 32):
                    d2 = ((x[:, None, :] - hc[None, h0:h0 + 32]) ** 2).sum(2)
                    m |= (d2 < rad[None, h0:h0 + 32] ** 2).any(1)
                p = levels[-1][m]
                oct_ = torch.tensor([[s & 1, (s >> 1) & 1, s >> 2] for s in range(8)], device=DEV)
                levels.append((2 * p[:, None, :] + oct_[None]).reshape(-1, 3))
        keys, lev, ctr = [], [], []
        for i, c in enumerate(levels):
            keys.append(_keys(base + i, c, self.table, self.marks))
            lev.append(torch.full((c.shape[0],), base + i, device=DEV))
            ctr.append(self._centres(base + i, c))
        keys, order = torch.sort(torch.cat(keys))
        self.keys, self.level, self.x = keys, torch.cat(lev)[order], torch.cat(ctr)[order]
        # the base field (trilinear) and the haloes (NFW, cut off at four r200)
        u = self.x * nbox - 0.5
        i0 = torch.floor(u)
        fr, i0 = u - i0, i0.long()
        val = torch.zeros((self.x.shape[0], 5), device=DEV, dtype=F64)
        for s in range(8):
            b = [(s >> d) & 1 for d in range(3)]
            idx = [(i0[:, d] + b[d]) % nbox for d in range(3)]
            wt = torch.ones_like(fr[:, 0])
            for d in range(3):
                wt = wt * (fr[:, d] if b[d] else 1 - fr[:, d])
            val += wt[:, None] * field[(idx[0] * nbox + idx[1]) * nbox + idx[2]]
        if hal is not None:
            hc, r200, rs, gm = hal
            for h in range(nh):
                cut = 4.0 * float(r200[h])
                at = torch.nonzero(((self.x - hc[h]).abs() < cut).all(1))[:, 0]
                dv = (self.x[at] - hc[h]) * LENGTH
                d = dv.norm(dim=1)
                rc = cut * LENGTH
                r = d.clamp(min=1e-3 * float(rs[h]))

                def phi(r):
                    return -gm[h] * torch.log1p(r / rs[h]) / r

                def dphi(r):
                    return gm[h] * (torch.log1p(r / rs[h]) / r ** 2 - 1.0 / (r * (rs[h] + r)))

                rct = torch.tensor(rc, device=DEV, dtype=F64)
                p = torch.where(d < rc, phi(r) - phi(rct) - (r - rct) * dphi(rct), 0.0)
                q = torch.where(d < rc, dphi(r) - dphi(rct), 0.0)
                val[at, 0] += p
                val[at, 1:4] += (q / d.clamp(min=1e-30))[:, None] * dv
                val[at, 4] -= p / (1e-5 * CLIGHT ** 2)
        zt = torch.from_numpy(np.stack([_chi, _z])).to(DEV)
        a = 1.0 / (1.0 + _interp(self.x.norm(dim=1) * LBOX, zt[0], zt[1]))
        ea = torch.sqrt(OM / a ** 3 + 1 - OM)
        dphidt = val[:, 0] * (1.0 - (OM / a ** 3 / ea ** 2) ** 0.55) * a * H0 * ea
        # rho phi dphidx dphidy dphidz a dphidt, as the records hold them
        self.f = torch.stack([val[:, 4], val[:, 0], val[:, 1], val[:, 2], val[:, 3], a, dphidt], 1).float()

    @staticmethod
    def _centres(L, c):
        return (c.to(F64) + 0.5) * (4.0 / 2 ** L) - 2.0

    def records(self):
        n = self.keys.shape[0]
        r = torch.zeros((n, 12), device=DEV, dtype=torch.int32)
        r[:, 2] = (self.keys & 0xffffffff).to(torch.int32)
        r[:, 3] = (self.keys >> 32).to(torch.int32)
        r[:, 4:11] = self.f[:, [6, 5, 2, 3, 4, 1, 0]].contiguous().view(torch.int32)
        return r.cpu().numpy().view(np.dtype((np.void, 48))).reshape(-1)

    def find(self, level, c):
        """Cells of exactly `level` at coordinates c, or -1."""
        side = (1 << level) if isinstance(level, int) else torch.ones_like(level) << level
        inside = ((c >= 0) & (c < (side if isinstance(level, int) else side[..., None]))).all(-1)
        k = _keys(level, torch.where(inside[..., None], c, 0), self.table, self.marks)
        i = torch.searchsorted(self.keys, k.contiguous()).clamp(max=self.keys.numel() - 1)
        return torch.where(inside & (self.keys[i] == k), i, -1)

    def coords(self, level, x):
        s = 2.0 ** (level - 2) if isinstance(level, int) else torch.pow(2.0, (level - 2).to(F64))[:, None]
        return torch.floor((x + 2.0) * s).long()

    def locate(self, x):
        """(deepest cell, its level) holding each point; -1 outside the cone."""
        cell = torch.full((x.shape[0],), -1, device=DEV)
        lev = torch.full((x.shape[0],), self.base, device=DEV)
        for L in range(self.base, self.top + 1):
            i = self.find(L, self.coords(L, x))
            lev = torch.where(i >= 0, L, lev)
            cell = torch.where(i >= 0, i, cell)
        return cell, lev

    def gather(self, order, x, fields, extra=None):
        """CIC (1) or TSC (2) of the cells' fields at points x in float64: all vertices of the
        located cell's level, else again at the level of the first coarser one; 0 where one is missing."""
        src = fields if extra is None else torch.cat([fields, extra], 1)
        out = torch.zeros((x.shape[0], src.shape[1]), device=DEV, dtype=F64)
        cell, lev = self.locate(x)
        todo = torch.nonzero(cell >= 0)[:, 0]
        o = torch.tensor([[a, b, c] for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)] if order == 2 else
                         [[v & 1, (v >> 1) & 1, v >> 2] for v in range(8)], device=DEV)
        for _ in range(self.top - self.base + 1):
            if not todo.numel():
                break
            p, L = x[todo], lev[todo]
            c = self.coords(L, p)
            fd = (p + 2.0) * torch.pow(2.0, (L - 2).to(F64))[:, None] - c - 0.5
            if order == 2:
                w3 = torch.stack([0.5 * (0.5 - fd) ** 2, 0.75 - fd ** 2, 0.5 * (0.5 + fd) ** 2], -1)
                w = (w3[:, 0, :, None, None] * w3[:, 1, None, :, None] * w3[:, 2, None, None, :]).reshape(-1, 27)
                nb = c[:, None, :] + o[None]
            else:
                side = torch.where(fd >= 0, 1, -1)
                nb = c[:, None, :] + o[None] * side[:, None, :]
                w = torch.where(o[None] == 1, fd.abs()[:, None, :], 1 - fd.abs()[:, None, :]).prod(-1)
            i = self.find(L[:, None].expand(-1, o.shape[0]), nb)
            full = (i >= 0).all(1)
            out[todo[full]] = (w[full][:, :, None] * src[i[full]].to(F64)).sum(1)
            rest = torch.nonzero(~full)[:, 0]
            if not rest.numel():
                break
            # the level at which the first missing vertex (CIC: the coarsest) has a cell
            first = (i[rest] < 0).to(torch.int32).argmax(1)
            cand = nb[rest] if order == 1 else nb[rest, first][:, None, :]
            have = i[rest] >= 0 if order == 1 else torch.zeros((rest.numel(), 1), dtype=torch.bool, device=DEV)
            up = torch.where(have, L[rest][:, None], -1)
            for k in range(1, self.top - self.base + 1):
                lk = (L[rest] - k).clamp(min=self.base)[:, None].expand(-1, cand.shape[1])
                sh = (L[rest][:, None] - lk)[..., None]
                hit = (self.find(lk, cand >> sh) >= 0) & (up < 0) & ((L[rest] - k) >= self.base)[:, None]
                up = torch.where(hit, lk, up)
            up = up.amin(1)
            ok = (up >= 0) & (up < L[rest])
            todo = todo[rest[ok]]
            lev[todo] = up[ok]
        return out


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _pkg():
    return importlib.import_module(PKG)


def _directions(case, seed, n):
    """A grid of directions over the cone in rows (the photon grid's order), shifted by the seed."""
    rng = np.random.default_rng(int(seed) + 5)
    side = int(math.ceil(math.sqrt(n)))
    j = rng.uniform(0.25, 0.75, 2)
    t = 0.96 * HALF * (2 * (np.arange(side)[:, None] + j[None, :]) / side - 1)
    ph, th = np.meshgrid(np.radians(t[:, 0]), np.pi / 2 + np.radians(t[:, 1]), indexing="ij")
    d = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], -1).reshape(-1, 3)
    return np.ascontiguousarray(d[:n])


def _pixels(case):
    """RING pixels of the cone about +x, in the map's order."""
    ns, n = case["nside"], case["n"]
    t = math.radians(0.96 * HALF)
    j = min(int(t / (math.pi / (2 * ns))) - 1, int(math.sqrt(n) / 2) + 1)
    rows = np.arange(2 * ns - n // (2 * j + 1) // 2 - 2, 4 * ns)
    cols = np.concatenate([np.arange(0, j + 1), np.arange(4 * ns - j, 4 * ns)])
    return np.ascontiguousarray((2 * ns * (ns - 1) + 4 * ns * (rows[:, None] - ns) + cols[None, :]).ravel()[:n].astype(np.int64))


def _surfaces(case):
    z = case["z"]
    return np.array([z * (k + 1) / case["planes"] for k in range(case["planes"])])


def _homogeneous(zs):
    t, a, _ = _cosmology()
    return np.array([(np.interp(-1.0 / (1 + z), -a, t), _chi_of_z(z), np.interp(-1.0 / (1 + z), -a, t), 1.0 / (1 + z), z)
                     for z in zs])


def _cell_velocities(cone):
    g = cone.f[:, 2:5].to(F64)
    v = -g / g.square().sum(1).mean().sqrt() * 1e-3
    return v.float()


VOBS = (6e-4, -3e-4, 2e-4)       # in units of c, as the cells' velocities
COMPONENTS = ["lensing", "dr", "dt", "isw", "dens", "deflection"]


def prepare(case, seed):
    pkg = _pkg()
    cone = Cone(case, seed)
    t, a, dadt = _cosmology()
    s = {"case": case, "pkg": pkg, "cosmo": pkg.Cosmology(t, a, dadt)}
    kind = case["kind"]
    if kind == "cells":
        s["rows"], s["cone"] = _cell_rows(case, cone, seed)
        return s
    s["tree"] = pkg.Octree.from_records(cone.records())
    if kind == "rays":
        launch = np.zeros((case["n"], 6))
        launch[:, 3:] = _directions(case, seed, case["n"])
        s["launch"] = launch
        if case["vel"]:
            s["tree"].set_velocity(_cell_velocities(cone).cpu().numpy())
        if case["device"]:
            capi = importlib.import_module(PKG + ".capi")
            n, npl = case["n"], case["planes"]
            s["capi"], s["lib"] = capi, pkg.library()
            s["dlaunch"] = torch.from_numpy(launch).to(DEV)
            s["dsteps"] = torch.zeros(n, dtype=torch.int64, device=DEV)
            s["dfinal"] = torch.zeros((n, capi.MPF_PHOTON_FIELDS), dtype=F64, device=DEV)
            s["dplanes"] = torch.zeros((n, npl, capi.MPF_PLANE_FIELDS), dtype=F64, device=DEV) if npl else None
            s["dstatus"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif kind == "maps":
        s["pixels"] = _pixels(case)
        s["surfaces"] = _surfaces(case)
        s["homogeneous"] = _homogeneous(s["surfaces"])
    elif kind == "catalogue":
        rng = np.random.default_rng(int(seed) + 9)
        n = case["n"]
        d = _chi_of_z(case["z"]) * rng.uniform(0.02, 1.0, n) ** (1 / 3)
        ph, th = np.radians(rng.uniform(-4.5, 4.5, n)), np.pi / 2 + np.radians(rng.uniform(-4.5, 4.5, n))
        src = np.zeros((n, 8))
        src[:, 0], src[:, 1], src[:, 2] = d * np.cos(ph) * np.sin(th), d * np.sin(ph) * np.sin(th), d * np.cos(th)
        src[:, 3:6] = rng.normal(0.0, 1e-3, (n, 3))
        src[:, 6], src[:, 7] = np.arange(n), 1.0
        s["sources"] = src
    elif kind == "bundles":
        rng = np.random.default_rng(int(seed) + 11)
        ph = np.zeros((case["n"], 6))
        d = _directions(case, seed, case["n"])
        ph[:, 3:] = d[rng.permutation(case["n"])]
        s["photons"], s["rotation"] = ph, rng.uniform(0.0, 2 * np.pi, case["n"])
    elif kind == "deposit":
        pos, vel = _particles(case, cone, seed)
        s["pos"], s["vel"] = pos.cpu().numpy(), vel.cpu().numpy()
    return s


def _particles(case, cone, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 3)
    nxt = torch.cat([cone.level[1:], torch.zeros(1, dtype=cone.level.dtype, device=DEV)])
    leaf = torch.nonzero(nxt <= cone.level)[:, 0]
    pick = leaf[torch.randint(0, leaf.numel(), (case["n"],), generator=g, device=DEV)]
    size = 4.0 / torch.pow(2.0, cone.level[pick].to(F64))
    pos = cone.x[pick] + (torch.rand((case["n"], 3), generator=g, device=DEV, dtype=F64) - 0.5) * size[:, None]
    vel = _cell_velocities(cone)[pick].to(F64) + 1e-4 * torch.randn((case["n"], 3), generator=g, device=DEV, dtype=F64)
    return pos.float(), vel.float()


def _cell_rows(case, cone, seed):
    """The cone's cells as the simulation writes them (level, centre, rho, phi, force, a; code units) in blocks of
    unsorted order; a fraction `dup` again at the next shell's time, a fraction `drop` of the refined cells lost."""
    g, gs = torch.Generator(device=DEV), torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 104729 + 1)
    gs.manual_seed(815)                  # which cells are there does not change with the seed
    a = cone.f[:, 5].to(F64)
    t = a * a * MPC / (HUB * 1e5)
    l = a * LBOX * MPC / HUB
    r = torch.zeros((cone.keys.numel(), 10), device=DEV, dtype=F64)
    r[:, 0] = (cone.level - 2).to(F64)
    r[:, 1:4] = cone.x
    r[:, 4] = cone.f[:, 0]
    r[:, 5] = cone.f[:, 1].to(F64) * (t / l) ** 2
    r[:, 6:9] = cone.f[:, 2:5].to(F64) / ((l / (t * t)) * (-a))[:, None]
    r[:, 9] = a
    if case["drop"] > 0:
        lost = (cone.level > cone.base) & (torch.rand(cone.level.shape, generator=gs, device=DEV) < case["drop"])
        r = r[~lost]
    if case["dup"] > 0:
        again = r[torch.rand(r.shape[0], generator=gs, device=DEV) < case["dup"]].clone()
        again[:, 9] *= 1.001
        again[:, 5] *= 1.0005
        r = torch.cat([r, again])
    nb = -(-r.shape[0] // 4096)
    at = (torch.randperm(nb, generator=g, device=DEV)[:, None] * 4096 + torch.arange(4096, device=DEV)[None]).reshape(-1)
    r = r[at[at < r.shape[0]]]
    xmax = _chi_of_z(case["z"]) * 1.02
    return r.float().cpu().numpy(), dict(cone_vertex=(0.0, 0.0, 0.0), cone_base=(xmax * 1.1, 0.0, 0.0),
                                         cone_angle=math.radians(1.2 * math.sqrt(2.0) * HALF), sphere_center=(0.0, 0.0, 0.0),
                                         sphere_radius=0.03)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, pkg, kind = s["case"], s["pkg"], s["case"]["kind"]
    if kind == "rays":
        pl = _surfaces(case) if case["planes"] else None
        kw = dict(nsteps=case["nsteps"], order=case["order"], stop="redshift", stop_value=case["z"], planes=pl,
                  jacobian=case["jac"], exact=case["exact"], vobs=VOBS if case["vel"] else (0.0, 0.0, 0.0))
        if not case["device"]:
            steps, final, planes, _ = pkg.propagate(s["tree"], s["cosmo"], s["launch"], LENGTH, **kw)
            return {"steps": steps, "final": final, "planes": planes}
        capi, n = s["capi"], case["n"]
        p, keep = capi.make_params(LENGTH, **kw)
        ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())
        capi.check(s["lib"].mpf_propagate_device(s["tree"]._h, s["cosmo"]._h, C.byref(p), n, ptr(s["dlaunch"]),
                                                 ptr(s["dsteps"]), ptr(s["dfinal"]), ptr(s["dplanes"]), ptr(s["dstatus"]),
                                                 C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"steps": s["dsteps"], "final": s["dfinal"], "planes": s["dplanes"]}
    if kind == "maps":
        kw = dict(jacobian="bundle", plane="sachs", stop_bundle="redshift", openingmin=6e-5) if case["bundle"] else {}
        return pkg.hmaps_fill(s["tree"], s["cosmo"], case["nside"], s["pixels"], s["surfaces"], s["homogeneous"], COMPONENTS,
                              LENGTH, nsteps=case["nsteps"], order=case["order"], **kw)
    if kind == "catalogue":
        return pkg.catalogue(s["tree"], s["cosmo"], s["sources"], LENGTH, HUB, mpc=MPC, cat_accuracy=1e-8,
                             nsteps=case["nsteps"], order=case["order"])[0]
    if kind == "bundles":
        sizes, traj = pkg.rays_propagate(s["tree"], s["cosmo"], s["photons"], LENGTH, case["count"], math.radians(0.01),
                                         rotation=s["rotation"], amin=0.0, nsteps=case["nsteps"], order=case["order"],
                                         capacity=_capacity(case))
        return {"sizes": sizes, "trajectories": traj}
    if kind == "cells":
        return pkg.cells_build(s["rows"], s["cosmo"], h=HUB, omegam=OM, lboxmpch=LBOX, mpc=MPC, order=case["order"],
                               **s["cone"])
    s["tree"].deposit_velocity(s["pos"], s["vel"], scheme=case["order"])
    v, rho = s["tree"].velocity()
    return {"velocity": v, "rho": rho}


def _capacity(case):
    """Trajectory points kept per ray: the path's base cells and a wide allowance for refined ones."""
    return int(_chi_of_z(case["z"]) * 1.1 * 2 ** (case["base"] - 2) * case["nsteps"] * 2 + 2500)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    # cells of the cone: the base volume, and the refined spheres of a few thousand cells a level
    xmax = _chi_of_z(case["z"]) * 1.02
    cells = (2 * math.tan(math.radians(HALF))) ** 2 * (xmax * 2 ** (case["base"] - 2) + 6) ** 3 / 3 * 1.3
    cells += case["halos"] * 8000.0 * (case["top"] - case["base"])
    kind, tsc = case["kind"], case["order"] == 2
    if kind == "cells":
        return {"bytes": cells * (1 + case["dup"]) * 40 + cells * 48, "flops": cells * 60}
    if kind == "deposit":
        lv = case["top"] - case["base"] + 1
        pairs = case["n"] * (27 if tsc else 8) * (1 + 0.5 * (lv - 1))
        return {"bytes": case["n"] * 24 + cells * (16 + 16 + 16), "flops": pairs * 10}
    steps = xmax * 2 ** (case["base"] - 2) * case["nsteps"] * (1.0 + 0.2 * (case["top"] - case["base"]))
    g = 27 if tsc else 8
    jac = {"rays": case.get("jac"), "maps": not case.get("bundle"), "catalogue": False, "bundles": False}[kind]
    per = 4 * g * 8 + g * 14 + (6 * 27 * 6 if jac else 0) + 300
    n = case["n"]
    rays = n * (5 if case.get("bundle") else 1) if kind == "maps" else n * 3 if kind == "catalogue" else \
        n * (case["count"] + 1) if kind == "bundles" else n
    out = {"rays": n * (48 + 8 + 224 + 160 * case.get("planes", 0)), "maps": n * (8 + 4 * 10 * case.get("planes", 0)),
           "catalogue": n * (64 + 128), "bundles": n * _capacity(case) * 232.0 if kind == "bundles" else 0}[kind]
    return {"bytes": cells * 48 + out, "flops": rays * steps * per}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
class Tracer:
    """The null-geodesic integration of the framework (fourth-order Runge-Kutta in the affine parameter, steps of a
    fraction of the local cell) with everything in float64, all rays at once."""

    def __init__(self, cone, case, vel=None):
        self.cone, self.case, self.vel = cone, case, vel
        t, a, dadt = _cosmology()
        self.t, self.a, self.dadt = (torch.from_numpy(v.copy()).to(DEV) for v in (t, a, dadt))
        self.f = cone.f.to(F64)

    def field(self, x):
        return self.cone.gather(self.case["order"], x, self.f, self.vel)

    def rhs(self, y):
        d = self.field(y[:, 2:5])
        k0, k = y[:, 5:6], y[:, 6:9]
        g, dt = d[:, 2:5], d[:, 6:7]
        gk = (g * k).sum(1, keepdim=True)
        dphidl = dt * k0 + gk
        dadt = _interp(y[:, 1], self.t, self.dadt)[:, None]
        hub = 2 * dadt / y[:, 0:1] * k0
        c2 = CLIGHT ** 2
        return torch.cat([k0 * dadt, k0, k / LENGTH, -hub * k0 - 2 / c2 * k0 * gk,
                          -hub * k + 2 / c2 * dphidl * k - 2 * g * k0 * k0], 1)

    def hessian(self, x, lev):
        h = torch.pow(2.0, (2 - lev).to(F64))
        e = torch.eye(3, device=DEV, dtype=F64)
        e = torch.cat([e, -e])[:, None, :] * h[None, :, None]
        g = self.cone.gather(2, (x[None] + e).reshape(-1, 3), self.f[:, 2:5]).reshape(2, 3, -1, 3)
        g = (g[0] - g[1]) / (2 * h)[None, :, None]
        dxx, dxy, dxz, dyy, dyz, dzz = g[0][:, 0], g[1][:, 0], g[2][:, 0], g[1][:, 1], g[2][:, 1], g[2][:, 2]
        rho, r = x[:, :2].norm(dim=1), x.norm(dim=1)
        cp, sp, ct, st = x[:, 0] / rho, x[:, 1] / rho, x[:, 2] / r, rho / r
        return torch.stack([sp * sp * dxx + cp * cp * dyy - 2 * sp * cp * dxy,
                            ct * cp * sp * (dyy - dxx) + (cp * cp - sp * sp) * ct * dxy + sp * st * dxz - cp * st * dyz,
                            (cp * ct) ** 2 * dxx + (sp * ct) ** 2 * dyy + st ** 2 * dzz + 2 * sp * cp * ct ** 2 * dxy
                            - 2 * sp * st * ct * dyz - 2 * cp * st * ct * dxz], 1)

    def run(self, direction, planes, stop, jac, vobs=(0.0, 0.0, 0.0)):
        n, c2 = direction.shape[0], CLIGHT ** 2
        z1 = torch.zeros((n, 1), device=DEV, dtype=F64)
        k = torch.from_numpy(direction).to(DEV)
        k = k / k.norm(dim=1, keepdim=True)
        x0 = torch.zeros((n, 3), device=DEV, dtype=F64)
        d = self.cone.gather(1, x0, self.f, self.vel)         # the origin is gathered with CIC
        ph = d[:, 1:2] / c2
        k = k * torch.sqrt(c2 * (1 + 2 * ph) / ((1 - 2 * ph) * (k * k).sum(1, keepdim=True)))
        a0 = _interp(z1[:, 0], self.t, self.a)[:, None]
        b = torch.cat([a0, z1, x0, 1 + z1, k], 1)
        vo = torch.tensor(vobs, device=DEV, dtype=F64)
        v0n = (vo * k).sum(1) / CLIGHT
        _, lev = self.cone.locate(x0)
        ratio = LENGTH / CLIGHT / self.case["nsteps"]
        dl = 4.0 / torch.pow(2.0, lev.to(F64)) * b[:, 0] ** 2 * ratio
        phi0, bf = d[:, 1] / c2, d
        # isw iswold chi lambda s red
        acc = torch.zeros((n, 6), device=DEV, dtype=F64)
        bdt = d[:, 6].clone()
        s1 = torch.zeros((3, n, 6), device=DEV, dtype=F64)    # Jacobian sums at the point and the two before it
        chi = torch.zeros((3, n), device=DEV, dtype=F64)
        npl = len(planes)
        rec = torch.zeros((n, npl, 20), device=DEV, dtype=F64)
        crossed = torch.zeros((n, npl), dtype=torch.bool, device=DEV)
        rmax = torch.full((n,), -math.inf, device=DEV, dtype=F64)
        idx = torch.zeros(n, device=DEV, dtype=F64)
        final = torch.zeros((n, 28), device=DEV, dtype=F64)
        on = torch.arange(n, device=DEV)
        for _ in range(4000):
            if not on.numel():
                break
            y, h = b[on], dl[on][:, None]
            k1 = self.rhs(y)
            k2 = self.rhs(y + h / 2 * k1)
            k3 = self.rhs(y + h / 2 * k2)
            k4 = self.rhs(y + h * k3)
            p = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            d = self.field(p[:, 2:5])
            _, lev = self.cone.locate(p[:, 2:5])
            inside = (d != 0).any(1)                         # a point outside the cone ends the ray before it
            if not bool(inside.all()):
                on, y, h, p, d, lev = (v[inside] for v in (on, y, h, p, d, lev))
            q = acc[on].clone()
            o = bf[on]
            q[:, 0] += (bdt[on] - d[:, 6]) * (p[:, 1] - y[:, 1]) / c2
            q[:, 1] -= 2 * (d[:, 1] - o[:, 1]) / c2 - ((o[:, 2:5] + d[:, 2:5]) * (p[:, 2:5] - y[:, 2:5])).sum(1) * LENGTH / c2
            q[:, 2] = p[:, 2:5].norm(dim=1)
            q[:, 3] += h[:, 0]
            q[:, 4] += (p[:, 2:5] - y[:, 2:5]).norm(dim=1)
            br = 1 + phi0[on] - d[:, 1] / c2
            if self.vel is not None:
                br = br + q[:, 0] + (d[:, 7:10] * p[:, 6:9]).sum(1) / (CLIGHT * p[:, 5]) - v0n[on]
            q[:, 5] = a0[on, 0] / p[:, 0] * br - 1
            idx[on] += 1
            chi[2, on], chi[1, on], chi[0, on] = chi[1, on], chi[0, on], q[:, 2]
            if jac:
                hs = self.hessian(p[:, 2:5], lev) * (q[:, 2] - acc[on, 2])[:, None]
                s1[2, on], s1[1, on] = s1[1, on], s1[0, on]
                s1[0, on] += torch.cat([q[:, 2:3] * hs, q[:, 2:3] ** 2 * hs], 1)
            for j in range(npl):
                m = (~crossed[on, j]) & (q[:, 5] > planes[j])
                if not bool(m.any()):
                    continue
                at = on[m]
                crossed[at, j] = True
                z0, zq = acc[at, 5], q[m, 5]
                f = (zq - planes[j]) / (zq - z0)

                def mix(u, v):
                    return u * f + v * (1 - f)

                px = torch.stack([mix(y[m, 2 + e], p[m, 2 + e]) for e in range(3)], 1)
                dist = px.norm(dim=1)
                r = rec[at, j]
                r[:, 0], r[:, 1], r[:, 2:5], r[:, 5] = idx[at] - 1, f, px, dist
                r[:, 9], r[:, 10], r[:, 11] = mix(y[m, 1], p[m, 1]), mix(y[m, 0], p[m, 0]), mix(z0, zq)
                for e, w in ((12, 2), (13, 3), (14, 4), (15, 0)):
                    r[:, e] = mix(acc[at, w], q[m, w])
                r[:, 16], r[:, 17] = mix(bf[at, 0], d[m, 0]), mix(bf[at, 1], d[m, 1])
                r[:, 18] = torch.where(torch.isinf(rmax[at]), 0.0, rmax[at])
                r[:, 19] = 1.0
                if jac:
                    use = torch.where(chi[0, at] <= dist, 0, torch.where(chi[1, at] <= dist, 1, 2))
                    sm = s1[use, at]
                    jj = (sm[:, :3] - sm[:, 3:] / dist[:, None]) * (2 * LENGTH / c2)
                    r[:, 6], r[:, 7], r[:, 8] = 1 - jj[:, 0], -jj[:, 1], 1 - jj[:, 2]
                rec[at, j] = r
            rmax[on] = torch.maximum(rmax[on], bf[on, 0])
            pk = (p[:, 6:9] ** 2).sum(1)
            g00 = c2 * (1 + 2 * d[:, 1] / c2) * p[:, 5] ** 2
            gkk = (1 - 2 * d[:, 1] / c2) * pk
            final[on] = torch.stack([*p.T, lev.to(F64), d[:, 5], d[:, 0], d[:, 1], d[:, 2], d[:, 3], d[:, 4], -d[:, 6],
                                     d[:, 6] * p[:, 5] + (d[:, 2:5] * p[:, 6:9]).sum(1), (d[:, 1] - bf[on, 1]) / h[:, 0],
                                     q[:, 5], p[:, 0] ** 2 * (gkk - g00), 1 - gkk / g00, q[:, 0], q[:, 1], q[:, 2], q[:, 3],
                                     q[:, 4], idx[on]], 1)
            b[on], bf[on], acc[on], bdt[on] = p, d, q, -d[:, 6]
            dl[on] = 4.0 / torch.pow(2.0, lev.to(F64)) * p[:, 0] ** 2 * ratio
            on = on[~(q[:, 5] > stop)]
        # a surface crossed on the way to the last point only is no surface of the map
        for j in range(npl):
            last = rec[:, j, 0] == 0
            rec[last, j, 19] = 0.0
        return final, rec


def exact(case, seed):
    kind = case["kind"]
    if kind == "deposit":
        cone = Cone(case, seed)
        return _deposit64(case, cone, *_particles(case, cone, seed))
    if kind == "cells":
        return None                      # bytes
    if kind in ("catalogue", "bundles") or case.get("bundle"):
        return None                      # a float64 run of all rays of all rounds or bundles takes minutes
    # the longest ray's steps, at about a hundredth of a second each
    steps = _chi_of_z(case["z"]) * 2 ** (case["base"] - 2) * case["nsteps"] * (1 + 4 * (case["top"] - case["base"]))
    if steps > 1000 or case["n"] * steps > 4.5e6:
        return None                      # over twenty seconds
    cone = Cone(case, seed)
    vel = _cell_velocities(cone) if case.get("vel") else None
    pl = _surfaces(case) if case["planes"] else np.zeros(0)
    tr = Tracer(cone, case, vel.to(F64) if vel is not None else None)
    if kind == "rays":
        final, rec = tr.run(_directions(case, seed, case["n"]), pl, case["z"], case["jac"], VOBS if case["vel"] else (0.0,) * 3)
        return {"steps": None, "final": final, "planes": rec if case["planes"] else None}
    ns, px = case["nside"], _pixels(case) - 2 * case["nside"] * (case["nside"] - 1)
    ring, j = ns + px // (4 * ns), px % (4 * ns)
    ct = 4.0 / 3.0 - 2.0 * ring / (3.0 * ns)
    ph, st = (j + 0.5 * ((ring - ns + 1) % 2)) * np.pi / (2 * ns), np.sqrt(1 - ct * ct)
    d = np.stack([st * np.cos(ph), st * np.sin(ph), ct], 1)
    _, r = tr.run(d, pl, float(pl[-1]), True)
    d, hom = torch.from_numpy(d).to(DEV), _homogeneous(pl)
    out = torch.zeros((len(pl), 10, case["n"]), device=DEV, dtype=F64)
    for k in range(len(pl)):
        a11, a12, a22, o = r[:, k, 6], r[:, k, 7], r[:, k, 8], r[:, k]
        rows = [1 - 0.5 * (a11 + a22), -0.5 * (a11 - a22), -a12, a11 * a22 - a12 ** 2, o[:, 12] / hom[k, 1] - 1,
                o[:, 9] / hom[k, 0] - 1, o[:, 15], o[:, 16],
                torch.atan2(d[:, 1], d[:, 0]) - torch.atan2(o[:, 3], o[:, 2]), torch.acos(d[:, 2]) - torch.acos(o[:, 4] / o[:, 5])]
        out[k] = torch.where(o[:, 19] > 0, torch.stack(rows), 0.0)
    return out


def _deposit64(case, cone, pos, vel):
    """Every particle's cloud at every level onto the cells there, then velocity = momentum / mass; a cell that no
    particle reaches has its parent's."""
    n = cone.keys.numel()
    m = torch.zeros(n, device=DEV, dtype=F64)
    p = torch.zeros((n, 3), device=DEV, dtype=F64)
    x, v = pos.to(F64), vel.to(F64)
    for L in range(cone.base, cone.top + 1):
        c = cone.coords(L, x)
        fd = (x + 2.0) * 2.0 ** (L - 2) - c - 0.5
        if case["order"] == 2:
            offs = [(a, b, e) for a in (-1, 0, 1) for b in (-1, 0, 1) for e in (-1, 0, 1)]
            w3 = torch.stack([0.5 * (0.5 - fd) ** 2, 0.75 - fd ** 2, 0.5 * (0.5 + fd) ** 2], -1)
        else:
            offs = [(s & 1, (s >> 1) & 1, s >> 2) for s in range(8)]
            w3 = torch.stack([1 - fd.abs(), fd.abs()], -1)
        side = torch.where(fd >= 0, 1, -1)
        for o in offs:
            ot = torch.tensor(o, device=DEV)
            q = [e + 1 for e in o] if case["order"] == 2 else o
            i = cone.find(L, c + ot * (1 if case["order"] == 2 else side))
            w = w3[:, 0, q[0]] * w3[:, 1, q[1]] * w3[:, 2, q[2]]
            hit = i >= 0
            m.index_add_(0, i[hit], w[hit])
            p.index_add_(0, i[hit], (w[:, None] * v)[hit])
    out = p / torch.where(m == 0, 1.0, m)[:, None]
    for L in range(cone.base + 1, cone.top + 1):
        at = torch.nonzero((cone.level == L) & (m.float().abs() < torch.finfo(torch.float32).tiny))[:, 0]
        up = cone.find(L - 1, cone.coords(L - 1, cone.x[at]))
        out[at[up >= 0]] = out[up[up >= 0]]
    return {"velocity": out, "rho": m}
