"""What users of this framework have it do, as measurable cases.

A user's program builds a structured or read mesh, hands it to a `Solver`,
sets it up and solves one or many load cases, either in one go (the
reference's own main program) or again and again against the resident
factors; a program with its own Krylov loop calls the dual operators.  (A `Server`
makes the calls of a mixed-form program for every request.)  The cases cover
those calls from the reference's default problem (eight subdomains of 5^3 elements, where latency
counts) to the 512-subdomain cube, with uniform and uneven slabs, both forms
(fp64 and mixed), the three preconditioners and one or several load cases.

Kinds of case:
  program  create, set_mesh, set_loads, setup, pcpg: a new problem end to end
  solve    new load cases against the resident factors (htf_solve)
  ops      one step of a caller's own dual iteration: P, F, P and the
           preconditioner on host vectors
  project  the projector on device vectors, on the caller's stream
"""
import math
import random

import numpy as np
import torch

import hfls_b200 as hb


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def _case(name, kind, clusters, subs, lo, hi, wseed, contrast=1.0, E=1.0, precision="fp64", pre="Dirichlet_explicit",
          nrhs=1, batch=32):
    """Slab widths (elements per subdomain and axis) are drawn from lo..hi."""
    d = {"name": name, "kind": kind, "cx": clusters[0], "cy": clusters[1], "cz": clusters[2], "sx": subs[0],
         "sy": subs[1], "sz": subs[2], "lo": lo, "hi": hi, "wseed": wseed, "E": E, "contrast": contrast,
         "precision": precision, "pre": pre, "nrhs": nrhs, "batch": batch}
    if name is None:
        del d["name"]
    return d


def listed():
    return [
        # the reference's own problem, solved again with new loads: latency
        _case("solve_reference", "solve", (1, 1, 1), (2, 2, 2), 5, 5, 0, E=2.1e5),
        # the same problem as the reference's main program runs it: everything from the mesh arrays to u
        _case("program_reference", "program", (1, 1, 1), (2, 2, 2), 5, 5, 0, E=2.1e5),
        # a caller's own dual iteration on a small uneven problem with the lumped preconditioner
        _case("ops_small_lumped", "ops", (2, 1, 1), (2, 2, 2), 3, 7, 1, contrast=10.0, pre="lumped"),
        # the same on 512 smaller subdomains, three vectors at once
        _case("ops_sub512", "ops", (2, 2, 2), (4, 4, 4), 4, 6, 0, contrast=10.0, nrhs=3),
        # the projector alone, on device vectors, between a caller's own kernels
        _case("project_device", "project", (2, 2, 2), (2, 2, 2), 4, 10, 2),
        # one load case on 64 subdomains of very different sizes (a mesh partitioned by geometry)
        _case("solve_uneven64", "solve", (2, 2, 2), (2, 2, 2), 4, 12, 0, contrast=10.0),
        # several load cases in full FP64 (a user who does not want the mixed form)
        _case("solve_fp64_loads8", "solve", (2, 2, 1), (2, 2, 2), 4, 9, 3, contrast=10.0, nrhs=8),
        # the storage-saving preconditioner, odd sizes
        _case("solve_implicit", "solve", (1, 2, 1), (3, 2, 2), 3, 8, 4, contrast=10.0, pre="Dirichlet_implicit"),
        # the batched mixed form, a full batch of load cases
        _case("batch_mixed32", "solve", (2, 2, 2), (2, 2, 2), 8, 8, 0, contrast=10.0, precision="mixed", nrhs=32),
        # a new small problem in the mixed form with a few load cases, as a server runs each request
        _case("program_mixed_loads5", "program", (2, 1, 1), (2, 2, 2), 4, 7, 5, contrast=10.0, precision="mixed",
              nrhs=5, batch=16),
        # a new uneven problem end to end: set-up dominates
        _case("program_uneven64", "program", (2, 2, 2), (2, 2, 2), 4, 12, 0, contrast=10.0),
        # the 512-subdomain cube end to end
        _case("program_cube512", "program", (2, 2, 2), (4, 4, 4), 8, 8, 0, contrast=10.0),
    ]


def draw(rng):
    """One more case of the same ranges: at most 64 subdomains of at most 12 elements per axis, and no more set-up
    work than 64 uneven subdomains take."""
    while True:
        c = _drawn(rng)
        if work(dict(c, kind="program", pre="Dirichlet_explicit", precision="fp64", nrhs=1))["flops"] < 1.2e12:
            return c


def _drawn(rng):
    kind = rng.choice(["solve", "solve", "solve", "program", "program", "ops", "ops", "project"])
    lo = rng.randint(2, 8)
    hi = min(12, lo + rng.randint(0, 6))
    clusters = tuple(rng.choice([1, 1, 2]) for _ in range(3))
    subs = [rng.choice([2, 2, 3]) for _ in range(3)]
    while clusters[0] * clusters[1] * clusters[2] * subs[0] * subs[1] * subs[2] > 64:
        subs[rng.randrange(3)] = 2
        clusters = tuple(rng.choice([1, 1, 2]) for _ in range(3))
    kw = {"contrast": rng.choice([1.0, 3.0, 10.0])}
    if kind == "solve":
        if rng.random() < 0.4:
            kw.update(precision="mixed", nrhs=rng.randint(1, 32), batch=rng.choice([16, 32]))
        else:
            kw.update(nrhs=int(round(math.exp(rng.uniform(0.0, math.log(12.0))))),
                      pre=rng.choice(["Dirichlet_explicit", "Dirichlet_explicit", "lumped", "Dirichlet_implicit"]))
    elif kind == "ops":
        # F on larger subdomains is not reproducible enough to be compared: its local inverses cancel in the
        # coarse correction, to about 1e-9
        lo, hi = min(lo, 4), min(hi, 6)
        kw.update(nrhs=rng.randint(1, 5), contrast=10.0,
                  pre=rng.choice(["Dirichlet_explicit", "lumped", "Dirichlet_implicit"]))
    elif kind == "program":
        if rng.random() < 0.3:
            kw.update(precision="mixed", batch=rng.choice([16, 32]))
        kw.update(pre=rng.choice(["Dirichlet_explicit", "lumped"]), nrhs=rng.randint(1, 3))
    return _case(None, kind, clusters, tuple(subs), lo, hi, rng.randrange(1 << 20), **kw)


# --------------------------------------------------------------------------
# meshes: a unit cube of hex8 elements cut into uneven slabs, as a user's own
# mesh generator would hand it over
# --------------------------------------------------------------------------
def _widths(case):
    r = random.Random(case["wseed"])
    return [[r.randint(case["lo"], case["hi"]) for _ in range(case["c" + a] * case["s" + a])] for a in "xyz"]


def _mesh(case, seed, jitter=0.1):
    """Arrays of one problem; jitter and materials from the seed."""
    w = _widths(case)
    rng = np.random.default_rng([int(seed), 1])
    ne = [sum(v) for v in w]
    nn = [n + 1 for n in ne]
    slab = [np.repeat(np.arange(len(v)), v) for v in w]
    bound = [np.concatenate([[0], np.cumsum(v)]) for v in w]
    k, j, i = np.meshgrid(*[np.arange(n) for n in reversed(nn)], indexing="ij")
    ijk = [i.ravel(), j.ravel(), k.ravel()]
    coords = np.stack([ijk[0] * (1.0 / ne[0]) - 0.5 + 0.5, ijk[1] * (1.0 / ne[1]) - 0.5 + 0.5, ijk[2] * (1.0 / ne[2])], 1)
    inner = np.ones(len(coords), bool)
    for a in range(3):
        inner &= (ijk[a] > 0) & (ijk[a] < ne[a])
    if jitter:
        coords[inner] += jitter * rng.uniform(-1.0, 1.0, (int(inner.sum()), 3)) / np.array(ne)
    ek, ej, ei = [v.ravel() for v in np.meshgrid(*[np.arange(n) for n in reversed(ne)], indexing="ij")]
    sy, sz = nn[0], nn[0] * nn[1]
    f0 = ei + ej * sy + ek * sz
    elems = np.stack([f0, f0 + 1, f0 + 1 + sy, f0 + sy, f0 + sz, f0 + 1 + sz, f0 + 1 + sy + sz, f0 + sy + sz], 1)
    g = [slab[0][ei], slab[1][ej], slab[2][ek]]
    S = [case["sx"], case["sy"], case["sz"]]
    cl = g[0] // S[0] + case["cx"] * (g[1] // S[1] + case["cy"] * (g[2] // S[2]))
    loc = g[0] % S[0] + S[0] * (g[1] % S[1] + S[1] * (g[2] % S[2]))
    per = S[0] * S[1] * S[2]
    nsub = per * case["cx"] * case["cy"] * case["cz"]
    E = case["E"] * np.exp(rng.uniform(0.0, 1.0, nsub) * math.log(case["contrast"]))
    dirichlet = (3 * np.flatnonzero(ijk[0] == 0)[:, None] + np.arange(3)).ravel()
    corner = []
    for kk in bound[2]:
        for jj in bound[1]:
            for ii in bound[0]:
                if ii in (0, ne[0]) and jj in (0, ne[1]) and kk in (0, ne[2]):
                    continue
                n = ii + sy * jj + sz * kk
                corner += [3 * n, 3 * n + 1, 3 * n + 2]
    return {"coords": coords, "elems": elems.astype(np.int32), "elem_sub": (cl * per + loc).astype(np.int32),
            "sub_cluster": (np.arange(nsub) // per).astype(np.int32), "E": E, "nu": np.full(nsub, 0.3),
            "dirichlet": dirichlet.astype(np.int32), "corner": np.array(corner, np.int32),
            "body": np.array([0.0, 0.0, -1.0]), "face": np.flatnonzero(ijk[0] == ne[0])}


def _user_mesh(m):
    return hb.Mesh(m["coords"], m["elems"], m["elem_sub"], m["sub_cluster"], m["E"], m["nu"], m["dirichlet"],
                   m["corner"], m["body"])


def _loads(case, m, seed):
    """Nodal forces on the face x = 1, one row per load case, of the size of the body force there."""
    rng = np.random.default_rng([int(seed), 2])
    n = case["nrhs"]
    f = np.zeros((n, len(m["coords"]), 3))
    f[:, m["face"], :] = rng.standard_normal((n, len(m["face"]), 3)) / len(m["face"])
    return f.reshape(n, -1)


def _options(case):
    o = {"typeBc": "cor", "max_iter": "1000", "preconditioner": case["pre"], "precision": case["precision"]}
    # displacements to about 1e-10 either way: the mixed form stops at a tenth of its eps_iter by itself
    o["eps_iter"] = "1e-9" if case["precision"] == "mixed" else "1e-10"
    if case["precision"] == "mixed":
        o["batch"] = str(case["batch"])
    return o


def _vectors(case, n_lambda, seed):
    return np.random.default_rng([int(seed), 3]).standard_normal((case["nrhs"], n_lambda))


# --------------------------------------------------------------------------
# the framework's part
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    m = _mesh(case, seed)
    mesh, opts = _user_mesh(m), _options(case)
    if kind == "program":
        return {"kind": kind, "mesh": mesh, "opts": opts, "f": _loads(case, m, seed)}
    s = hb.Solver(opts)
    s.set_mesh(mesh)
    s.setup()
    if kind == "solve":
        return {"kind": kind, "solver": s, "f": _loads(case, m, seed), "u": np.zeros((case["nrhs"], 3 * mesh.n_nodes))}
    x = _vectors(case, s.n_lambda(), seed)
    if kind == "ops":
        return {"kind": kind, "solver": s, "x": x}
    xd = torch.from_numpy(x[0]).cuda()
    return {"kind": kind, "solver": s, "x": xd, "y": torch.empty_like(xd)}


def run(state):
    kind = state["kind"]
    if kind == "program":
        s = hb.Solver(state["opts"])
        s.set_mesh(state["mesh"])
        s.set_loads(state["f"])
        s.setup()
        u, _ = s.pcpg()
        s.close()
        return {"u": u}
    s = state["solver"]
    if kind == "solve":
        u, _ = s.solve(state["f"], u=state["u"])
        return {"u": u}
    if kind == "ops":
        Px = s.projection(state["x"])
        PFPx = s.projection(s.mult_Ff(Px))
        return {"Px": Px, "PFPx": PFPx, "MPx": s.preconditioning(Px)}
    s.projection_noalloc(state["x"].data_ptr(), state["y"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return {"Px": state["y"]}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
# PCPG iterations that the path's rule takes on these problems (they depend on
# the material contrast and the stopping rule, little on the size)
def _iterations(case):
    base = {"Dirichlet_explicit": 80, "Dirichlet_implicit": 80, "lumped": 120}[case["pre"]]
    return base if case["contrast"] == 1.0 else int(1.2 * base)


def _sizes(case):
    """(DOFs, interface and clamped DOFs) of every subdomain, and the number of dual rows."""
    w = _widths(case)
    out, rows = [], 0
    for k, wz in enumerate(w[2]):
        for j, wy in enumerate(w[1]):
            for i, wx in enumerate(w[0]):
                tot = (wx + 1) * (wy + 1) * (wz + 1)
                inn = (wx + 1 - 1 - (i + 1 < len(w[0])))
                inn *= (wy + 1 - (j > 0) - (j + 1 < len(w[1]))) * (wz + 1 - (k > 0) - (k + 1 < len(w[2])))
                out.append((3 * tot, 3 * (tot - max(inn, 0))))
    rows = sum(nb for _, nb in out) // 2
    return out, rows


def work(case):
    kind, nrhs = case["kind"], case["nrhs"]
    subs, rows = _sizes(case)
    if kind == "project":
        return {"bytes": rows * (8.0 * (1 + 1 + 12) + 8.0), "flops": 4.0 * rows * 12}
    passes = 2 if case["pre"] == "Dirichlet_implicit" else 1
    entry = 4.0 if case["precision"] == "mixed" else 8.0
    tri = sum(nb * (nb + 1) / 2 for _, nb in subs)
    full = sum(n * (n + 1) / 2 for n, _ in subs)
    if kind == "ops":
        return {"bytes": (1 + passes) * 8.0 * tri + 8.0 * 4 * rows * nrhs, "flops": 4.0 * nrhs * (1 + passes) * tri}
    its = _iterations(case)
    # the matrices once per iteration, the factor once for the start and twice for the displacements, nodal loads in
    # and displacements out
    by = its * (1 + passes) * entry * tri + 3 * 8.0 * full + 2 * 8.0 * nrhs * sum(n for n, _ in subs)
    fl = nrhs * (its * (1 + passes) * 4.0 * tri + 3 * 4.0 * full)
    if kind == "program":
        # Cholesky of every K_i and F_i = (L_bb L_bb^T)^{-1}
        fl += sum(n ** 3 / 3.0 + 2.0 * nb ** 3 / 3.0 for n, nb in subs)
        by += 8.0 * (2 * full + 2 * tri)
    return {"bytes": by, "flops": fl}


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _element_matrices(m):
    """Stiffness (ne x 24 x 24) and body-force load (ne x 24) of the hex8 elements, DOF order 3 node + component."""
    dev = _dev()
    X = torch.from_numpy(m["coords"]).to(dev)[torch.from_numpy(m["elems"]).long().to(dev)]        # ne 8 3
    E = torch.from_numpy(m["E"]).to(dev)[torch.from_numpy(m["elem_sub"]).long().to(dev)]
    nu = 0.3
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    sg = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                       [-1, 1, 1]], dtype=torch.float64, device=dev)
    ne = len(X)
    K = torch.zeros(ne, 8, 3, 8, 3, dtype=torch.float64, device=dev)
    F = torch.zeros(ne, 8, 3, dtype=torch.float64, device=dev)
    body = torch.from_numpy(m["body"]).to(dev)
    for p in sg / math.sqrt(3.0):
        t = 1 + sg * p                                                                              # 8 3
        N = t.prod(1) / 8
        dN = torch.stack([sg[:, 0] * t[:, 1] * t[:, 2], sg[:, 1] * t[:, 0] * t[:, 2], sg[:, 2] * t[:, 0] * t[:, 1]], 1) / 8
        J = torch.einsum("eai,aj->eij", X, dN)
        det = torch.linalg.det(J)
        G = torch.einsum("aj,eji->eai", dN, torch.linalg.inv(J))
        s = torch.einsum("eai,ebj->eaibj", G, G)
        d = torch.einsum("eak,ebk->eab", G, G)
        wl, wm = (lam * det)[:, None, None, None, None], (mu * det)[:, None, None, None, None]
        K += wl * s + wm * s.permute(0, 1, 4, 3, 2)
        for c in range(3):
            K[:, :, c, :, c] += (mu * det)[:, None, None] * d
        F += det[:, None, None] * N[None, :, None] * body
    return K.reshape(ne, 24, 24), F.reshape(ne, 24)


def _elem_dofs(m):
    return (3 * m["elems"].astype(np.int64)[:, :, None] + np.arange(3)).reshape(-1, 24)


def _displacements(m, f):
    """K u = body force + f with u = 0 on the clamped face, by conjugate gradients on the whole mesh."""
    dev = _dev()
    Ke, Fe = _element_matrices(m)
    dof = torch.from_numpy(_elem_dofs(m)).to(dev)
    n = 3 * len(m["coords"])
    free = torch.ones(n, dtype=torch.float64, device=dev)
    free[torch.from_numpy(m["dirichlet"]).long().to(dev)] = 0.0
    b = torch.from_numpy(f).to(dev).clone()
    b += torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, dof.reshape(-1), Fe.reshape(-1))
    b *= free
    diag = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, dof.reshape(-1),
                                                                      Ke.diagonal(dim1=1, dim2=2).reshape(-1))
    nr, flat = len(b), dof.reshape(-1)

    def mul(p):
        y = torch.einsum("eij,rej->rei", Ke, p[:, dof]).reshape(nr, -1)
        return torch.zeros_like(p).index_add_(1, flat, y) * free

    x = torch.zeros_like(b)
    r = b.clone()
    for _ in range(2):                              # a second solve from the true residual
        p = torch.zeros_like(b)
        rz_old, goal = None, 1e-14 * b.norm(dim=1)
        for it in range(3000):
            z = r / diag
            rz = (r * z).sum(1)
            p = z if rz_old is None else z + (rz / rz_old.clamp_min(1e-300))[:, None] * p
            Ap = mul(p)
            a = (rz / (p * Ap).sum(1).clamp_min(1e-300))[:, None]
            x += a * p
            r = r - a * Ap
            rz_old = rz
            if it % 20 == 19 and bool((r.norm(dim=1) < goal).all()):
                break
        r = b - mul(x)
    return x.cpu().numpy()


def _dual(m):
    """Rows of Bf: ((subdomain, DOF), (subdomain, DOF) or None) in the framework's order, and their weights."""
    dof, nsub = _elem_dofs(m), len(m["sub_cluster"])
    ds = np.unique(dof.reshape(-1) * nsub + np.repeat(m["elem_sub"].astype(np.int64), 24))
    g, d = ds // nsub, ds % nsub
    clamped = np.zeros(3 * len(m["coords"]), bool)
    clamped[m["dirichlet"]] = True
    start = np.searchsorted(g, np.arange(3 * len(m["coords"]) + 1))
    cnt = np.diff(start)
    a, b, at, wt = [], [], [], []
    for c in np.unique(cnt[cnt >= 2]):              # DOFs shared by c subdomains
        gs = np.flatnonzero((cnt == c) & ~clamped)
        for p in range(c):
            for q in range(p + 1, c):
                a.append(d[start[gs] + p])
                b.append(d[start[gs] + q])
                at.append(gs)
                wt.append(np.full(len(gs), 1.0 / c))
    a, b, at, wt = [np.concatenate(v) for v in (a, b, at, wt)]
    o = np.lexsort((b, at, a))
    a, b, at, wt = a[o], b[o], at[o], wt[o]
    on = clamped[g]
    o = np.lexsort((g[on], d[on]))
    a = np.concatenate([a, d[on][o]])
    b = np.concatenate([b, np.full(int(on.sum()), -1)])
    at = np.concatenate([at, g[on][o]])
    return a, b, at, np.concatenate([wt, np.ones(int(on.sum()))])


def _rigid(m, dofs):
    """The six rigid modes at the given DOFs (n x 6)."""
    X, c = m["coords"][dofs // 3], dofs % 3
    R = np.zeros((len(dofs), 6))
    R[np.arange(len(dofs)), c] = 1.0
    R[c == 0, 3], R[c == 1, 3] = -X[c == 0, 1], X[c == 1, 0]
    R[c == 0, 4], R[c == 2, 4] = -X[c == 0, 2], X[c == 2, 0]
    R[c == 1, 5], R[c == 2, 5] = -X[c == 1, 2], X[c == 2, 1]
    return R


def _projector(m, dual):
    dev = _dev()
    a, b, at, _ = dual
    ncl = int(m["sub_cluster"].max()) + 1
    R = _rigid(m, at)
    G = np.zeros((len(a), ncl, 6))
    r = np.arange(len(a))
    np.add.at(G, (r, m["sub_cluster"][a]), R)
    two = b >= 0
    np.add.at(G, (r[two], m["sub_cluster"][b[two]]), -R[two])
    Q = torch.linalg.qr(torch.from_numpy(G.reshape(len(a), -1)).to(dev)).Q
    return lambda x: x - (Q @ (Q.T @ x.T)).T


def _operators(case, m, x):
    dev = _dev()
    dual = _dual(m)
    a, b, at, wt = dual
    P = _projector(m, dual)
    Px = P(torch.from_numpy(x).to(dev))
    w = torch.from_numpy(wt).to(dev)
    Ke, _ = _element_matrices(m)
    dof, nrhs = _elem_dofs(m), len(x)
    nsub, cl = len(m["sub_cluster"]), m["sub_cluster"]
    corner = np.zeros(3 * len(m["coords"]), bool)
    corner[m["corner"]] = True
    subs = []
    for d in range(nsub):
        es = np.flatnonzero(m["elem_sub"] == d)
        l2g, inv = np.unique(dof[es].reshape(-1), return_inverse=True)
        n = len(l2g)
        K = torch.zeros(n * n, dtype=torch.float64, device=dev)
        inv = torch.from_numpy(inv.reshape(-1, 24)).to(dev)
        K.index_add_(0, (inv[:, :, None] * n + inv[:, None, :]).reshape(-1), Ke[torch.from_numpy(es).to(dev)].reshape(-1))
        R = torch.linalg.qr(torch.from_numpy(_rigid(m, l2g)).to(dev)).Q
        ra, rb = np.flatnonzero(a == d), np.flatnonzero(b == d)
        rows = torch.from_numpy(np.concatenate([ra, rb])).to(dev)
        pos = torch.from_numpy(np.searchsorted(l2g, np.concatenate([at[ra], at[rb]]))).to(dev)
        sign = torch.cat([torch.ones(len(ra)), -torch.ones(len(rb))]).double().to(dev)
        subs.append({"l2g": l2g, "K": K.reshape(n, n), "R": R, "rows": rows, "pos": pos, "sign": sign})
    # corner rows of every cluster: a shared corner DOF of d against the next subdomain of the cluster that has it
    ncl = int(cl.max()) + 1
    bc = [[] for _ in range(nsub)]
    owner = {}
    for d in range(nsub):
        for g in subs[d]["l2g"][corner[subs[d]["l2g"]]]:
            owner.setdefault(int(g), []).append(d)
    ncr = [0] * ncl
    for g in sorted(owner):
        for c in range(ncl):
            ds = [d for d in owner[g] if cl[d] == c]
            for p, q in zip(ds, ds[1:]):
                bc[p].append((ncr[c], g, 1.0))
                bc[q].append((ncr[c], g, -1.0))
                ncr[c] += 1
    F, M = torch.zeros_like(Px), torch.zeros_like(Px)
    for c in range(ncl):
        ds = [d for d in range(nsub) if cl[d] == c]
        n0 = ncr[c]
        A = torch.zeros(n0 + 6 * len(ds), n0 + 6 * len(ds), dtype=torch.float64, device=dev)
        rhs = torch.zeros(n0 + 6 * len(ds), nrhs, dtype=torch.float64, device=dev)
        keep = []
        for k, d in enumerate(ds):
            s = subs[d]
            n = len(s["l2g"])
            rho = s["K"].diagonal().mean()
            L = torch.linalg.cholesky(s["K"] + rho * s["R"] @ s["R"].T)
            f = torch.zeros(n, nrhs, dtype=torch.float64, device=dev).index_add_(
                0, s["pos"], (s["sign"] * Px[:, s["rows"]]).T.contiguous())
            B = torch.zeros(n0, n, dtype=torch.float64, device=dev)
            for r, g, v in bc[d]:
                B[r, int(np.searchsorted(s["l2g"], g))] = v
            KB, Kf, i6 = torch.cholesky_solve(B.T.contiguous(), L), torch.cholesky_solve(f, L), n0 + 6 * k
            A[:n0, :n0] += B @ KB
            A[:n0, i6:i6 + 6] = -B @ s["R"]
            A[i6:i6 + 6, :n0] = A[:n0, i6:i6 + 6].T
            rhs[:n0] += B @ Kf
            rhs[i6:i6 + 6] = -s["R"].T @ f
            keep.append((d, KB, Kf, i6))
            # preconditioner
            bs = torch.unique(s["pos"])
            xw = torch.zeros(n, nrhs, dtype=torch.float64, device=dev).index_add_(
                0, s["pos"], (s["sign"] * (w * Px)[:, s["rows"]]).T.contiguous())
            y = torch.zeros_like(xw)
            y[bs] = s["K"][bs][:, bs] @ xw[bs]
            if case["pre"] != "lumped":
                ins = torch.ones(n, dtype=torch.bool, device=dev)
                ins[bs] = False
                ii = ins.nonzero()[:, 0]
                if len(ii):
                    Li = torch.linalg.cholesky(s["K"][ii][:, ii])
                    y[bs] -= s["K"][bs][:, ii] @ torch.cholesky_solve(s["K"][ii][:, bs] @ xw[bs], Li)
            M.index_add_(1, s["rows"], s["sign"] * y[s["pos"]].T)
        # singular by the cluster's rigid modes: add their projector in alpha space
        H = torch.zeros(n0 + 6 * len(ds), 6, dtype=torch.float64, device=dev)
        for d, _, _, i6 in keep:
            H[i6:i6 + 6] = subs[d]["R"].T @ torch.from_numpy(_rigid(m, subs[d]["l2g"])).to(dev)
        H = torch.linalg.qr(H).Q
        sol = torch.linalg.solve(A + A.abs().max() * H @ H.T, rhs)
        for d, KB, Kf, i6 in keep:
            s = subs[d]
            u = Kf - KB @ sol[:n0] + s["R"] @ sol[i6:i6 + 6]
            F.index_add_(1, s["rows"], s["sign"] * u[s["pos"]].T)
    return {"Px": Px.cpu().numpy(), "PFPx": P(F).cpu().numpy(), "MPx": (w * M).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    m = _mesh(case, seed)
    if kind in ("solve", "program"):
        return {"u": _displacements(m, _loads(case, m, seed))}
    dual = _dual(m)
    x = _vectors(case, len(dual[0]), seed)
    if kind == "project":
        return {"Px": _projector(m, dual)(torch.from_numpy(x).to(_dev()))[0]}
    return _operators(case, m, x)
