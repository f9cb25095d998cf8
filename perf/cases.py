"""The work whose speed matters, as measurable cases.

A case is a dict of plain values: a geometry (point dipoles in a cube, or the
RWG functions of a meshed sphere), the operator's options and the call a user's
program makes on it.  `listed()` names the ones that stand for the range,
`draw(rng)` gives more of it; `prepare` builds what the program holds before the
call (the set-up operator, its input vectors, a stream), `run` makes one call,
`work` counts what the call cannot do without, and `exact` evaluates every
interaction directly in 64 bits where that is affordable.

Calls:
  device    y = A x on device vectors, on the program's own stream
  mapped    y = A x on page-locked host vectors (the end-to-end call)
  adjoint   y = A^H x on host vectors, with diagonal loads (gradients)
  multi     Y = A X for nrhs device vectors at once
  batch     count independent problems of uneven size in one launch
  solve     GMRES(restart), a fixed number of iterations, host vectors
  flexible  FGMRES with an inner solver on the complex-float far field
  solve_multi  GMRES on nrhs right-hand sides at once
"""
import functools
import math

import numpy as np
import torch

from mlfma_b200 import MLFMA, Batch, inputs

K = 2.0 * math.pi  # wavelength 1: every length is in wavelengths
CK = complex(0.0, -299792458.0 * 1.256637e-6 / (4.0 * math.pi)) * K  # the operator is C k Z


def _dipoles(name, n, side, call, **kw):
    c = dict(name=name, geometry="dipoles", n=n, side=side, leaf=64, call=call, precision=0, ref_compat=0,
             self_terms=1, tune=False, nrhs=1, count=1, iters=0, restart=0, inner=0)
    c.update(kw)
    return c


def _sphere(name, level, radius, call, **kw):
    c = dict(name=name, geometry="sphere", level=level, radius=radius, leaf=54, call=call, precision=0, ref_compat=0,
             self_terms=0, tune=False, nrhs=1, count=1, iters=0, restart=0, inner=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest operator with a far field: launches and latency
        _dipoles("dipoles 600", 600, 4.0, "device"),
        # dipoles in a 4-wavelength cube, plain FP64, 0.5-wavelength leaves
        _dipoles("dipoles 8192", 8192, 4.0, "device"),
        # uneven independent dipole problems in one launch, complex-float far field
        _dipoles("batch of 8 dipole problems", 30000, 6.0, "batch", precision=1, count=8),
        # many right-hand sides, an odd number, complex-float far field, ragged size
        _dipoles("dipoles 12347 x 17 rhs mixed", 12347, 3.7, "multi", precision=1, nrhs=17),
        # a small mesh: the adjoint product of a gradient computation, loads on
        _sphere("sphere 7680 adjoint", 4, 1.13, "adjoint"),
        # the r = 2 sphere, 30,720 RWGs: the reference's operator, tuned once
        _sphere("sphere 30720", 5, 2.0, "device", ref_compat=1, tune=True),
        # the same product end to end on pinned host vectors
        _sphere("sphere 30720 mapped", 5, 2.0, "mapped"),
        # ... with the complex-float far field
        _sphere("sphere 30720 mixed", 5, 2.0, "device", precision=1),
        # ... on 64 incident waves at once
        _sphere("sphere 30720 x 64 rhs", 5, 2.0, "multi", nrhs=64),
        # one GMRES(50) cycle of the EFIE solve
        _sphere("sphere 30720 gmres", 5, 2.0, "solve", self_terms=1, iters=50, restart=50),
        # two outer steps of the mixed flexible solve, ragged radius
        _sphere("sphere 30720 fgmres", 5, 1.83, "flexible", precision=1, self_terms=1, iters=50, restart=30, inner=25),
        # the large problem: r = 8 sphere, 491,520 RWGs, seven levels
        _sphere("sphere 491520 mixed", 7, 8.0, "device", precision=1, self_terms=1),
    ]


def draw(rng):
    """One more case of the ranges above."""
    def log_int(a, b):
        return int(math.exp(rng.uniform(math.log(a), math.log(b))))

    prec = rng.randrange(2)
    call = rng.choice(["device", "device", "device", "mapped", "adjoint", "multi", "multi", "batch", "solve",
                       "flexible", "solve_multi"])
    kw = dict(precision=prec)
    if call == "multi":
        kw["nrhs"] = rng.randint(2, 64)
    if call == "batch":
        kw.update(count=rng.randint(2, 10))
    if call == "solve":
        kw.update(iters=rng.randint(10, 50), restart=50, self_terms=1)
    if call == "solve_multi":
        kw.update(nrhs=rng.randint(2, 16), iters=rng.randint(4, 10), restart=50, self_terms=1)
    if call == "flexible":
        kw.update(precision=1, iters=50, restart=30, inner=25, self_terms=1)
    if call == "batch" or rng.random() < 0.4:
        n = log_int(600, 10000 if call in ("multi", "solve", "flexible", "solve_multi") else 50000)
        # a cube that keeps the mean leaf around half a wavelength or less
        side = round(rng.uniform(0.8, 1.4) * 4.0 * (n / 8192.0) ** (1.0 / 3.0), 3)
        kw.setdefault("self_terms", 1)
        kw["leaf"] = rng.choice([24, 32, 48, 64])
        c = _dipoles("", max(n, 2500) if call == "batch" else n, side, call, **kw)
    else:
        level = rng.choice([3, 4, 5, 6] if call in ("device", "mapped") else
                           [3, 4] if call == "solve_multi" else [3, 4, 5])
        radius = round(2.0 ** (level - 4) * rng.uniform(0.7, 1.3), 3)
        c = _sphere("", level, radius, call, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------- geometry

@functools.lru_cache(maxsize=8)
def _icosphere(level):
    """Unit icosphere by repeated midpoint subdivision: vertices, faces and the
    RWG list (edge vertices, the two triangles)."""
    t = (1.0 + 5.0 ** 0.5) / 2.0
    V = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                  (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], dtype=np.float64)
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    F = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
                  (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5),
                  (2, 4, 11), (6, 2, 10), (8, 6, 7), (9, 8, 1)], dtype=np.int64)

    def edges(F):
        e = np.sort(np.concatenate([F[:, [0, 1]], F[:, [1, 2]], F[:, [2, 0]]]), axis=1)
        return np.unique(e[:, 0] * (1 << 32) + e[:, 1], return_inverse=True)

    for _ in range(level):
        key, inv = edges(F)
        m = V[key >> 32] + V[key & 0xffffffff]
        nf = len(F)
        ab, bc, ca = (inv[i * nf:(i + 1) * nf] + len(V) for i in range(3))
        V = np.concatenate([V, m / np.linalg.norm(m, axis=1, keepdims=True)])
        a, b, c = F.T
        F = np.stack([np.stack(q, 1) for q in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))], 1).reshape(-1, 3)
    key, inv = edges(F)
    order = np.argsort(inv, kind="stable")  # the two faces of each edge, in face order
    tri = (order % len(F)).reshape(-1, 2)
    tri.sort(axis=1)
    E = np.concatenate([np.stack([key >> 32, key & 0xffffffff], 1), tri], axis=1)
    return V, F.astype(np.int32), np.ascontiguousarray(E.astype(np.int32))


def _mesh(case):
    V, F, E = _icosphere(case["level"])
    return inputs.RWGMesh(vertices=V * case["radius"], faces=F, rwgs=E)


def _clouds(case):
    """The dipole problems of a case: one, or count of uneven size (the largest
    first, log-uniform down to a fifteenth of it)."""
    out = []
    for i in range(case["count"]):
        n = int(case["n"] * 15.0 ** (-i / max(1, case["count"] - 1)))
        side = case["side"] * (n / case["n"]) ** (1.0 / 3.0)
        out.append((inputs.make_dipoles(n, side=side, seed=100 + i), side))
    return out


def _wave(seed):
    rng = np.random.default_rng(seed)
    k = rng.standard_normal(3)
    k /= np.linalg.norm(k)
    p = np.cross(k, rng.standard_normal(3))
    p /= np.linalg.norm(p)
    return inputs.PlaneWave(amplitude=1.0, pol=tuple(p), khat=tuple(k), wavenum=K)


def _options(case):
    return dict(max_node_srcs=case["leaf"], precision=case["precision"], ref_compat=case["ref_compat"],
                self_terms=case["self_terms"], max_rhs=case["nrhs"])


def _operators(case):
    pw = inputs.PlaneWave()
    if case["geometry"] == "sphere":
        return [MLFMA.rwg(_mesh(case), pw, root_leng=2.0 * case["radius"], **_options(case)).setup()]
    return [MLFMA.dipoles(d, pw, root_leng=side, **_options(case)).setup() for d, side in _clouds(case)]


def _total(case):
    if case["geometry"] == "sphere":
        return 30 * 4 ** case["level"]
    return sum(d.n for d, _ in _clouds(case))


def _host_vector(n, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def _vectors(case, seed):
    """The call's input vectors, on the host: (nrhs, n) complex."""
    n = _total(case)
    return np.stack([_host_vector(n, 1000 * seed + r) for r in range(case["nrhs"])])


def _loads(case):
    """Diagonal impedance loads of the adjoint call."""
    rng = np.random.default_rng(77)
    n = _total(case)
    return 1e-3 * (rng.uniform(0.0, 50.0, n) + 1j * rng.uniform(-20.0, 20.0, n))


# ---------------------------------------------------------------- the calls

_streams = {}


def _stream():
    """The program's stream: one, as its products depend on one another."""
    dev = torch.cuda.current_device()
    if dev not in _streams:
        _streams[dev] = torch.cuda.Stream()
    return _streams[dev]


def prepare(case, seed):
    ops = _operators(case)
    call = case["call"]
    st = dict(case=case, ops=ops, op=ops[0])
    if case["tune"]:
        ops[0].autotune()
    if call in ("solve", "flexible", "solve_multi"):
        waves = [_wave(1000 * seed + r) for r in range(case["nrhs"])]
        st["b"] = np.stack([ops[0].rhs_planewave(w) for w in waves])
        return st
    x = _vectors(case, seed)
    if call == "adjoint":
        ops[0].set_loads(_loads(case))
        st["x"] = x[0]
        return st
    x = torch.from_numpy(x if call == "multi" else x[0])
    if call == "mapped":
        st["x"] = x.pin_memory()
        st["y"] = torch.zeros_like(x).pin_memory()
        return st
    st["x"] = x.cuda()
    st["y"] = torch.zeros_like(st["x"])
    st["stream"] = _stream()
    if call == "batch":
        st["batch"] = Batch(ops)
    return st


def run(st):
    case, op, call = st["case"], st["op"], st["case"]["call"]
    if call == "device":
        op.matvec_device(st["x"].data_ptr(), st["y"].data_ptr(), False, st["stream"].cuda_stream)
        return st["y"]
    if call == "mapped":
        op.matvec_mapped(st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if call == "adjoint":
        return op.matvec_adjoint(st["x"])
    if call == "multi":
        op.matvec_multi_device(case["nrhs"], st["x"].data_ptr(), st["y"].data_ptr(), False, st["stream"].cuda_stream)
        return st["y"]
    if call == "batch":
        st["batch"].matvec_device(st["x"].data_ptr(), st["y"].data_ptr(), st["stream"].cuda_stream)
        return st["y"]
    # a fixed number of iterations: the tolerance is never met
    if call == "solve":
        x, info = op.solve(st["b"][0], max_iter=case["iters"], tol=1e-14, restart=case["restart"], ref_givens=False)
        return x, info.residual
    if call == "flexible":
        x, info = op.solve(st["b"][0], max_iter=case["iters"], tol=1e-14, restart=case["restart"], flexible=True,
                           inner_iters=case["inner"])
        return x, info.residual
    x, _ = op.solve_multi(st["b"], max_iter=case["iters"], tol=1e-14, restart=case["restart"])
    return x


# ---------------------------------------------------------------- work

@functools.lru_cache(maxsize=64)
def _sizes(key):
    """What the plan of a case's operators holds, summed: stored near-field
    entries, pattern values, list-2 values and level values (box-directions)."""
    case = dict(key)
    case.update(nrhs=1)
    pw = inputs.PlaneWave()
    if case["geometry"] == "sphere":
        ops = [MLFMA.rwg(_mesh(case), pw, root_leng=2.0 * case["radius"], **_options(case))]
    else:
        ops = [MLFMA.dipoles(d, pw, root_leng=side, **_options(case)) for d, side in _clouds(case)]
    near = patterns = values = tables = pairs = 0.0
    for op in ops:
        s = op.stats()
        near += s["near_entries"]
        patterns += 2.0 * s["pattern_elems"]
        boxes = 0
        for level in range(2, s["max_level"] + 1):
            g = op.level_info(level)
            nb = op.level_boxes(level).shape[0]
            ndir = g["nth"] * g["nph"]
            values += 2.0 * nb * ndir
            tables += 316.0 * ndir
            boxes += nb
            pairs += 2.0 * nb * ndir * s["list2"]
        pairs /= max(1, boxes)
        op.close()
    return near, patterns, values, tables, pairs


def work(case):
    """Bytes: each operator array read once per product (stored near-field
    entries, radiation patterns for aggregation and for disaggregation, transfer
    functions), outgoing and local patterns of every level written and read
    once, vectors in and out; a Krylov step reads its basis twice.  Flops: 8 per
    complex multiply-add of those entries, 24 taps per interpolated value."""
    near, patterns, values, tables, pairs = _sizes(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    n, r = float(_total(case)), case["nrhs"]
    cval = 16.0 if case["precision"] == 0 else 8.0
    half = 1.0 if case["precision"] == 0 else 0.5  # conjugate symmetry of a complex-float pattern
    matrix = near * 16.0 + 2.0 * patterns * cval * half + tables * cval
    vectors = 4.0 * values * cval + 2.0 * n * 16.0
    flops = 8.0 * (2.0 * near + 2.0 * patterns + pairs) + 4.0 * 2.0 * 24.0 * values
    products = max(1, case["iters"])
    basis = products * products * n * 16.0 * r if case["call"].startswith("solve") else 0.0
    return {"bytes": products * (matrix + r * vectors) + basis, "flops": products * r * flops + basis}


# ---------------------------------------------------------------- in 64 bits

# 7-point rule of a triangle: barycentric coordinates, weight
_RULE = [((1 / 3, 1 / 3, 1 / 3), 0.1125)] + \
    [(p, 0.066197076394253) for p in [(0.059715871789770, 0.470142064105115, 0.470142064105115),
                                      (0.470142064105115, 0.059715871789770, 0.470142064105115),
                                      (0.470142064105115, 0.470142064105115, 0.059715871789770)]] + \
    [(p, 0.0629695902724135) for p in [(0.797426985353087, 0.101286507323456, 0.101286507323456),
                                       (0.101286507323456, 0.797426985353087, 0.101286507323456),
                                       (0.101286507323456, 0.101286507323456, 0.797426985353087)]]


def _field(pos, cur, group, rows=None):
    """E[i] = sum_j G(r_i - r_j) J_j over points of other groups, G the dyadic
    Green's function e^{ikR}/R [(1 + i/kR - 1/k2R2) I - (1 + 3i/kR - 3/k2R2) RR].
    pos (p, 3), cur (p, 3, r) complex, group (p,) ids."""
    p, nr = pos.shape[0], cur.shape[2]
    out = torch.zeros_like(cur)
    step = max(1, int(6e7) // p)
    for i0 in range(0, p, step):
        d = [pos[i0:i0 + step, a, None] - pos[None, :, a] for a in range(3)]
        other = group[i0:i0 + step, None] != group[None, :]
        R = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        R = torch.where(other, R, torch.ones_like(R))
        inv = 1.0 / (K * R)
        g = torch.polar(other / R, K * R)
        A = g * torch.complex(1.0 - inv * inv, inv)
        B = g * torch.complex(1.0 - 3.0 * inv * inv, 3.0 * inv) / (R * R)
        E = torch.zeros(3, d[0].shape[0], nr, dtype=cur.dtype, device=cur.device)
        for a in range(3):
            E[a] += A @ cur[:, a]
            Ba = B * d[a]
            for b in range(3):
                E[a] -= (Ba * d[b]) @ cur[:, b]
        out[i0:i0 + step] = E.permute(1, 0, 2)
    return out


def _dipole_product(pos, mom, x, unit_diagonal):
    """Z x for unit dipoles; x (n, r)."""
    pos = torch.from_numpy(pos).cuda()
    ph = torch.from_numpy(mom / np.linalg.norm(mom, axis=1, keepdims=True)).cuda()
    E = _field(pos, ph[:, :, None] * x[:, None, :], torch.arange(len(pos), device=x.device))
    y = (ph[:, :, None] * E).sum(1)
    return y + x if unit_diagonal else y


def _rwg_product(mesh, x):
    """Z x for RWG functions by the 7-point rule on every pair of distinct
    triangles, an RWG's own two triangles left out; x (n, r)."""
    V = torch.from_numpy(mesh.vertices).cuda()
    F = torch.from_numpy(mesh.faces.astype(np.int64)).cuda()
    E = torch.from_numpy(mesh.rwgs.astype(np.int64)).cuda()
    bary = torch.tensor([b for b, _ in _RULE], dtype=torch.float64, device=V.device)
    w = torch.tensor([v for _, v in _RULE], dtype=torch.float64, device=V.device)
    nq, nf, nr = len(w), len(F), x.shape[1]
    q = torch.einsum("qv,fvc->fqc", bary, V[F])  # (f, q, 3)
    leng = (V[E[:, 0]] - V[E[:, 1]]).norm(dim=1)
    J = torch.zeros(nf, nq, 3, nr, dtype=x.dtype, device=x.device)
    basis = []
    for t in range(2):
        tri = E[:, 2 + t]
        fv = F[tri]
        free = V[fv.sum(1) - E[:, 0] - E[:, 1]]  # the vertex off the edge
        f = (1.0 - 2.0 * t) * leng[:, None, None] * w[None, :, None] * (q[tri] - free[:, None, :])  # (n, q, 3)
        basis.append((tri, f))
        J.index_add_(0, tri, f[..., None] * x[:, None, None, :])
    group = torch.arange(nf, device=x.device).repeat_interleave(nq)
    Ef = _field(q.reshape(-1, 3), J.reshape(-1, 3, nr), group).reshape(nf, nq, 3, nr)
    y = sum((f[..., None] * Ef[tri]).sum((1, 2)) for tri, f in basis)
    # an RWG's two triangles do not meet each other in its own entry
    (t0, f0), (t1, f1) = basis
    d = q[t0][:, :, None, :] - q[t1][:, None, :, :]
    R = d.norm(dim=-1)
    inv = 1.0 / (K * R)
    g = torch.polar(1.0 / R, K * R)
    uv = torch.einsum("npc,nqc->npq", f0, f1)
    urv = torch.einsum("npc,npqc->npq", f0, d) * torch.einsum("nqc,npqc->npq", f1, d) / (R * R)
    own = (g * (torch.complex(1.0 - inv * inv, inv) * uv - torch.complex(1.0 - 3.0 * inv * inv, 3.0 * inv) * urv))
    return y - 2.0 * own.sum((1, 2))[:, None] * x


def exact(case, seed):
    call = case["call"]
    if call in ("solve", "flexible", "solve_multi"):
        return None
    if case["geometry"] == "sphere" and (case["self_terms"] or case["level"] > 5):
        return None
    x = torch.from_numpy(_vectors(case, seed).T.copy()).cuda()  # (n, r)
    if call == "adjoint":  # A is complex-symmetric: A^H x = conj(A conj(x))
        x = x.conj().resolve_conj()
    if case["geometry"] == "sphere":
        y = _rwg_product(_mesh(case), x)
    else:
        y, at = [], 0
        for d, _ in _clouds(case):
            y.append(_dipole_product(d.pos, d.mom, x[at:at + d.n], case["self_terms"]))
            at += d.n
        y = torch.cat(y)
    y = CK * y
    if call == "adjoint":
        z = torch.from_numpy(_loads(case)).cuda()
        return (y + z[:, None] * x).conj().resolve_conj()[:, 0].cpu().numpy()
    if call == "multi":
        return y.T.contiguous()
    return y[:, 0].contiguous()
