"""Workloads of a CheFSI subspace iteration on one GPU, through skgemm's public calls.

What a real-space DFT solver asks of the library, call by call: the overlap
S = Psi^T Psi, the projected Hamiltonian Hs = Psi^T (H Psi), the rotation
Psi' = Psi Q, the producer of H Psi, batches of k-points, and the reference's
own blocking host calls. Grid sizes are cubes between 24^3 and 64^3 or the
10^4 .. 4*10^5 points of the serving range, state counts 32 .. 2048.

A case is a dict of plain values; `prepare` builds what a solver already holds
(packed operands, plan, projector set), `run` is one pass, `exact` the same
result in plain 64-bit torch.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "stream-k-gemm_b200"))
import skgemm  # noqa: E402

# 12th-order central second differences, radius 6 (the stencil's radius), for
# -1/2 nabla^2 at a grid spacing of 0.4.
_W = [-5369.0 / 1800.0, 12.0 / 7.0, -15.0 / 56.0, 10.0 / 189.0, -1.0 / 112.0, 2.0 / 1925.0,
      -1.0 / 16632.0]
_COEF = [-0.5 * w / 0.16 for w in _W]
_DV = 0.064
_PRECISION = {"native": skgemm.PREC_NATIVE, "ozaki": skgemm.PREC_OZAKI_I8}


def listed():
    return [
        # The smallest call of the serving range: one overlap matrix of a small
        # molecule, where launch latency counts.
        {"name": "syrk_small", "kind": "single", "op": "syrk", "precision": "native",
         "nd": 10000, "nb": 32, "nn": 32},
        # A plain dense row-major product, not a tile multiple (the reference's
        # own known-answer size).
        {"name": "gemm_dense_1000", "kind": "dense", "m": 1000, "n": 1000, "k": 1000},
        # A small cell, native precision: S, Hs and the rotation from band-packed
        # Psi, as a solver's inner loop issues them.
        {"name": "step_native_24", "kind": "step", "precision": "native", "layout": "band",
         "nd": 13824, "nb": 128},
        # The 48^3 x 512 configuration in native precision, the rotation from
        # the reference's grid-packed layout.
        {"name": "step_native_48", "kind": "step", "precision": "native", "layout": "grid",
         "nd": 110592, "nb": 512},
        # An ordinary cell on the split path, band-packed rotation, a state
        # count that is no multiple of the tiles.
        {"name": "step_ozaki_32", "kind": "step", "precision": "ozaki", "layout": "band",
         "nd": 32768, "nb": 336},
        # The 48^3 x 512 configuration on the split path (the benchmark's step).
        {"name": "step_ozaki_48", "kind": "step", "precision": "ozaki", "layout": "grid",
         "nd": 110592, "nb": 512},
        # The largest: 64^3 grid points, 1024 states, band-packed.
        {"name": "step_ozaki_64", "kind": "step", "precision": "ozaki", "layout": "band",
         "nd": 262144, "nb": 1024},
        # S and Hs together on an odd grid and an odd state count.
        {"name": "pair_ozaki_ragged", "kind": "pair", "precision": "ozaki", "nd": 42875,
         "nb": 333},
        # One product between two different blocks of states (a rectangular
        # result), split path, called alone as the reference's callers do.
        {"name": "gemm_ozaki_rect", "kind": "single", "op": "gemm", "precision": "ozaki",
         "nd": 91125, "nb": 500, "nn": 264},
        # 24 k-points of uneven size in one planned, graph-captured launch.
        {"name": "batch_kpoints", "kind": "batch", "count": 24, "mix": 7, "grid_max": 48,
         "nb_max": 512},
        # H Psi of the 48^3 x 512 configuration: halo, stencil, 64 atoms.
        {"name": "hpsi_48", "kind": "hpsi", "ni": 48, "nj": 48, "nk": 48, "nb": 512,
         "out_tile": 32, "atoms": 64, "radius": 5.75, "ncol": 16},
        # The reference's blocking call on host memory.
        {"name": "host_gemm", "kind": "host", "nd": 13824, "nb": 256},
    ]


_MOST = 262144 * 1024 ** 2  # nd * nb^2 of the largest listed case


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["single", "single", "dense", "step", "step", "step", "pair", "batch",
                       "hpsi", "host"])
    if kind == "single":
        op = rng.choice(["syrk", "gemm"])
        nd, nb = int(_log(rng, 1e4, 2.6e5)), int(_log(rng, 32, 1024))
        nn = nb if op == "syrk" else int(_log(rng, 32, 1024))
        return {"kind": kind, "op": op, "precision": rng.choice(["native", "ozaki"]), "nd": nd,
                "nb": nb, "nn": nn}
    if kind == "dense":
        return {"kind": kind, "m": int(_log(rng, 100, 3000)), "n": int(_log(rng, 100, 3000)),
                "k": int(_log(rng, 100, 3000))}
    if kind == "step":
        nb = 16 * max(2, round(_log(rng, 32, 2048) / 16))
        nd = 16 * round(_log(rng, 1e4, min(2.6e5, max(1.1e4, _MOST / nb ** 2))) / 16)
        return {"kind": kind, "precision": rng.choice(["native", "ozaki", "ozaki"]),
                "layout": rng.choice(["band", "grid"]), "nd": nd, "nb": nb}
    if kind == "pair":
        return {"kind": kind, "precision": rng.choice(["native", "ozaki"]),
                "nd": int(_log(rng, 1e4, 2e5)), "nb": int(_log(rng, 48, 900))}
    if kind == "batch":
        return {"kind": kind, "count": rng.randrange(4, 29), "mix": rng.randrange(1 << 20),
                "grid_max": rng.choice([32, 40, 48]), "nb_max": rng.choice([256, 384, 512])}
    if kind == "hpsi":
        ni, nj, nk = (rng.randrange(20, 57) for _ in range(3))
        return {"kind": kind, "ni": ni, "nj": nj, "nk": nk,
                "nb": int(_log(rng, 24, min(512, 5.6e7 / (ni * nj * nk)))),
                "out_tile": rng.choice([16, 32]), "atoms": rng.randrange(4, 65),
                "radius": round(rng.uniform(3.0, 6.0), 2), "ncol": rng.choice([4, 8, 9, 16])}
    return {"kind": kind, "nd": int(_log(rng, 4096, 4e4)), "nb": int(_log(rng, 32, 256))}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _packed(nd, nb, t, g, scale):
    """Random states in the packed-t layout [ceil(nb/t)][nd][t]; lanes past nb are zero."""
    x = torch.randn((nb + t - 1) // t, nd, t, dtype=torch.float64, device="cuda", generator=g)
    x *= scale
    if nb % t:
        x[-1, :, nb % t:] = 0.0
    return x


def _dense(x, nb):
    """[ceil(nb/t)][nd][t] -> (nd, nb)."""
    return x.permute(1, 0, 2).reshape(x.shape[1], -1)[:, :nb]


def _zeros(*shape):
    return torch.zeros(*shape, dtype=torch.float64, device="cuda")


def _mix(case):
    """The k-points of a batch: (grid points, states) of each."""
    r = random.Random(case["mix"])
    grids = [n for n in (24, 32, 40, 48) if n <= case["grid_max"]]
    return [(r.choice(grids) ** 3, int(_log(r, 64, case["nb_max"]))) for _ in range(case["count"])]


def _projectors(case, seed):
    """One ball of grid points per atom, its part inside the cell and its
    periodic images' part as two projectors that share the atom's columns."""
    ni, nj, nk = case["ni"], case["nj"], case["nk"]
    rng = np.random.default_rng(seed)
    m = int(math.ceil(case["radius"]))
    d = np.arange(-m, m + 1)
    dz, dy, dx = (a.ravel() for a in np.meshgrid(d, d, d, indexing="ij"))
    sets = {k: [] for k in ("nrow", "ncol", "atom", "index")}
    offsets = []
    for a in range(case["atoms"]):
        c = rng.uniform(0, 1, 3) * (ni, nj, nk)
        o = np.floor(c).astype(int)
        f = c - o
        ball = (dx - f[0]) ** 2 + (dy - f[1]) ** 2 + (dz - f[2]) ** 2 <= case["radius"] ** 2
        x, y, z = o[0] + dx[ball], o[1] + dy[ball], o[2] + dz[ball]
        inside = (x >= 0) & (x < ni) & (y >= 0) & (y < nj) & (z >= 0) & (z < nk)
        index = (x % ni) + ni * (y % nj) + ni * nj * (z % nk)
        for part in (inside, ~inside):
            if part.any():
                sets["nrow"].append(int(part.sum()))
                sets["ncol"].append(case["ncol"])
                sets["atom"].append(a + 1)
                sets["index"].append(index[part])
                offsets.append(a * case["ncol"])
    offsets.append(case["atoms"] * case["ncol"])
    chi = [rng.uniform(-1, 1, (case["ncol"], n)) for n in sets["nrow"]]  # column-major rows
    gamma = rng.uniform(-0.5, 0.5, (len(chi), case["ncol"]))
    return sets, offsets, chi, gamma


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        a = torch.rand(k, m, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        b = torch.rand(k, n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        return {"case": case, "a": a, "b": b, "d": _zeros(m, n)}
    if kind == "batch":
        pts, items = [], []
        for nd, nb in _mix(case):
            psi = _packed(nd, nb, 16, g, nd ** -0.5)
            hpsi = _packed(nd, nb, 32, g, nd ** -0.5)
            s, h = _zeros(nb, nb), _zeros(nb, nb)
            items.append(skgemm.batch_item(skgemm.OP_SYRK_PACKED, nb, nb, nd, psi, None, s, nb))
            items.append(skgemm.batch_item(skgemm.OP_GEMM_PACKED, nb, nb, nd, psi, hpsi, h, nb))
            pts.append((psi, hpsi, s, h))
        return {"case": case, "pts": pts, "plan": skgemm.Plan(items)}
    if kind == "hpsi":
        ni, nj, nk, nb, t = (case[x] for x in ("ni", "nj", "nk", "nb", "out_tile"))
        k = ni * nj * nk
        sets, offsets, chi, gamma = _projectors(case, seed)
        vnl = skgemm.NlocProjector(sets["nrow"], sets["ncol"], sets["atom"], offsets,
                                   np.concatenate(sets["index"]),
                                   np.concatenate([c.ravel() for c in chi]), gamma.ravel(), k)
        return {"case": case, "vnl": vnl, "psi": _packed(k, nb, 16, g, k ** -0.5),
                "ext": _zeros((nb + 15) // 16, nk + 12, nj + 12, ni + 12, 16),
                "pot": torch.rand(k, dtype=torch.float64, device="cuda", generator=g) - 1.0,
                "out": _zeros((nb + t - 1) // t, k, t)}
    if kind == "host":
        nd, nb = case["nd"], case["nb"]
        psi = _packed(nd, nb, 16, g, nd ** -0.5).cpu().numpy()
        hpsi = _packed(nd, nb, 32, g, nd ** -0.5).cpu().numpy()
        return {"case": case, "psi": psi, "hpsi": hpsi, "d": np.zeros((nb, nb))}
    nd, nb = case["nd"], case["nb"]
    st = {"case": case, "psi": _packed(nd, nb, 16, g, nd ** -0.5)}
    if kind == "single":
        st["b"] = st["psi"] if case["op"] == "syrk" else _packed(nd, case["nn"], 32, g, nd ** -0.5)
        st["d"] = _zeros(nb, case["nn"])
        return st
    st["hpsi"] = _packed(nd, nb, 32, g, nd ** -0.5)
    st["s"], st["hs"] = _zeros(nb, nb), _zeros(nb, nb)
    if kind == "step":
        st["q"] = torch.rand(nb, nb, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        st["rot"] = _zeros(nb // 16, nd, 16)
        if case["layout"] == "grid":
            st["grid"] = _dense(st["psi"], nb).reshape(-1, 16, nb).transpose(1, 2).contiguous()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        skgemm.dgemm_dev(m, n, k, st["a"], m, st["b"], n, st["d"], n)
        return st["d"]
    if kind == "batch":
        st["plan"].run()
        return [p[2:] for p in st["pts"]]
    if kind == "hpsi":
        ni, nj, nk, nb, t = (case[x] for x in ("ni", "nj", "nk", "nb", "out_tile"))
        skgemm.halo_periodic_dev(ni, nj, nk, nb, st["psi"], st["ext"])
        skgemm.stencil_ext_dev(ni, nj, nk, nb, st["ext"], st["pot"], _COEF, _COEF, _COEF,
                               3 * _COEF[0], st["out"], t)
        st["vnl"].apply(nb, _DV, st["psi"], st["out"], t)
        return st["out"]
    if kind == "host":
        nb = case["nb"]
        skgemm.gemm.compute_packed(nb, nb, case["nd"], st["psi"], st["hpsi"], st["d"])
        return st["d"]
    nd, nb, prec = case["nd"], case["nb"], _PRECISION[case["precision"]]
    if kind == "single":
        if case["op"] == "syrk":
            skgemm.dsyrk_packed_dev(nd, nb, st["psi"], st["d"], precision=prec)
        else:
            skgemm.dgemm_packed_dev(nb, case["nn"], nd, st["psi"], st["b"], st["d"], alpha=0.5,
                                    gamma=1e-3, precision=prec)
        return st["d"]
    skgemm.dsubspace_packed_dev(nd, nb, st["psi"], st["hpsi"], st["s"], st["hs"], precision=prec)
    if kind == "pair":
        return {"s": st["s"], "hs": st["hs"]}
    if case["layout"] == "grid":
        skgemm.drot_dev(nd, nb, st["grid"], st["q"], st["rot"], precision=prec)
    else:
        skgemm.drot_band_dev(nd, nb, st["psi"], st["q"], st["rot"], precision=prec)
    return {"s": st["s"], "hs": st["hs"], "rot": st["rot"]}


def work(case):
    kind = case["kind"]
    if kind == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8 * (m * k + k * n + m * n), "flops": 2 * m * n * k}
    if kind == "batch":
        mix = _mix(case)
        return {"bytes": sum(8 * (2 * nd * nb + nb * nb * 3 // 2) for nd, nb in mix),
                "flops": sum(nb * (nb + 1) * nd + 2 * nb * nb * nd for nd, nb in mix)}
    if kind == "hpsi":
        k, nb = case["ni"] * case["nj"] * case["nk"], case["nb"]
        rows = case["atoms"] * 4 / 3 * math.pi * case["radius"] ** 3
        return {"bytes": 8 * (2 * k * nb + k + rows * case["ncol"]),
                "flops": (55 * k + 4 * rows * case["ncol"]) * nb}
    nd, nb = case["nd"], case["nb"]
    if kind == "host":
        return {"bytes": 8 * (2 * nd * nb + nb * nb), "flops": 2 * nb * nb * nd}
    if kind == "single":
        nn = case["nn"]
        if case["op"] == "syrk":
            return {"bytes": 8 * (nd * nb + nb * nb // 2), "flops": nb * (nb + 1) * nd}
        return {"bytes": 8 * (nd * (nb + nn) + nb * nn), "flops": 2 * nb * nn * nd}
    w = {"bytes": 8 * (2 * nd * nb + nb * nb * 3 // 2),
         "flops": nb * (nb + 1) * nd + 2 * nb * nb * nd}
    if kind == "step":
        w["bytes"] += 8 * (2 * nd * nb + nb * nb)
        w["flops"] += 2 * nb * nb * nd
    return w


def _exact_hpsi(case, seed):
    ni, nj, nk, nb, t = (case[x] for x in ("ni", "nj", "nk", "nb", "out_tile"))
    k = ni * nj * nk
    g = _gen(seed)
    psi16 = _packed(k, nb, 16, g, k ** -0.5)
    pot = torch.rand(k, dtype=torch.float64, device="cuda", generator=g) - 1.0
    psi = _dense(psi16, nb).t().reshape(nb, nk, nj, ni).contiguous()
    out = psi * (pot.reshape(nk, nj, ni) + 3 * _COEF[0])
    for r in range(1, 7):
        for axis in (3, 2, 1):
            out += _COEF[r] * (torch.roll(psi, r, axis) + torch.roll(psi, -r, axis))
    psi, out = psi.reshape(nb, k), out.reshape(nb, k)
    sets, offsets, chi, gamma = _projectors(case, seed)
    parts = [(torch.from_numpy(i).cuda(), torch.from_numpy(c).cuda())
             for i, c in zip(sets["index"], chi)]
    coef = {}
    for p, (index, c) in enumerate(parts):
        a = sets["atom"][p]
        if a not in coef:
            coef[a] = [torch.from_numpy(gamma[p]).cuda(), 0.0]
        coef[a][1] = coef[a][1] + _DV * (psi[:, index] @ c.t())
    for p, (index, c) in enumerate(parts):
        gam, s = coef[sets["atom"][p]]
        out.index_add_(1, index, (s * gam) @ c)
    full = _zeros((nb + t - 1) // t * t, k)
    full[:nb] = out
    return full.reshape(-1, t, k).permute(0, 2, 1).contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind == "hpsi":
        return _exact_hpsi(case, seed)
    if kind == "host":
        g = _gen(seed)
        nd, nb = case["nd"], case["nb"]
        psi = _dense(_packed(nd, nb, 16, g, nd ** -0.5), nb)
        return (psi.t() @ _dense(_packed(nd, nb, 32, g, nd ** -0.5), nb)).cpu().numpy()
    if kind == "batch":
        g = _gen(seed)
        out = []
        for nd, nb in _mix(case):
            psi = _dense(_packed(nd, nb, 16, g, nd ** -0.5), nb)
            hpsi = _dense(_packed(nd, nb, 32, g, nd ** -0.5), nb)
            out.append((torch.tril(psi.t() @ psi), psi.t() @ hpsi))
        return out
    st = prepare(case, seed)
    if kind == "dense":
        return st["a"].t() @ st["b"]
    nb = case["nb"]
    psi = _dense(st["psi"], nb)
    if kind == "single":
        if case["op"] == "syrk":  # column-major upper triangle: row-major lower
            return torch.tril(psi.t() @ psi)
        return 0.5 * (psi.t() @ _dense(st["b"], case["nn"])) + 1e-3
    out = {"s": torch.tril(psi.t() @ psi), "hs": psi.t() @ _dense(st["hpsi"], nb)}
    if kind == "step":
        rot = psi @ st["q"]
        out["rot"] = rot.reshape(case["nd"], nb // 16, 16).permute(1, 0, 2).contiguous()
    return out
