"""The work that users of this framework have it do, as measurable cases.

Three kinds, each through a public entry point:

``march``  one network: ``Engine.run_net`` (every region the level set crosses,
           every face polygon), ``am_combine_mesh`` and ``am_get_mesh`` (the
           welded mesh into host arrays), on an engine and into arrays that the
           program keeps; the arrays hold more than the mesh, zeros behind it.  The three precisions
           a caller can choose are float64 (the reference's default dtype),
           float32 and mixed (tensor-core composition, FP64 vertices).
``batch``  several networks, or several boxes of one network, marched at once
           with ``engine.run_batch``, then each one's mesh.
``rows``   the constraint rows of given activation states, composed into the
           caller's buffers by ``am_compose_rows_noalloc``.

Networks are the seeded geometric initialisations of the benchmark
configurations ("net": the initialisation's seed); prepare()'s seed makes a
snapshot of the network, every parameter moved by a thousandth, and the seed
points, as a program has that meshes a network again while it trains.  Their
regions number about N^2 (unperturbed) or half of that, N the number of hidden
units.
"""
import ctypes
import math

import numpy as np
import torch

from analyticmesh_gb300 import _lib, engine, utils, workloads

# regions of a marching per (hidden units)^2
DENSITY = {"plain": 1.0, "perturbed": 0.5}


def listed():
    return [
        # the smallest call: the polytope example, in the reference's default precision
        {"name": "polytope14_f64", "kind": "march", "widths": "14", "polytope": True, "form": "float64",
         "seeds": 128},
        # a toy network, meshed again after every few training steps
        {"name": "mlp32x2_mixed", "kind": "march", "net": 7, "widths": "32,32", "form": "mixed", "seeds": 128},
        # a small shape network in plain float32
        {"name": "mlp64x3_f32", "kind": "march", "net": 12, "widths": "64,64,64", "form": "float32", "perturb": 0.01,
         "seeds": 1024},
        # the sphere configuration in each precision
        {"name": "sphere128x4_f32", "kind": "march", "net": 1, "widths": "128,128,128,128",
         "form": "float32", "seeds": 1024},
        {"name": "sphere128x4_f64", "kind": "march", "net": 1, "widths": "128,128,128,128",
         "form": "float64", "seeds": 1024},
        {"name": "sphere128x4_mixed", "kind": "march", "net": 1, "widths": "128,128,128,128",
         "form": "mixed", "seeds": 1024},
        # ragged widths, the input added into a layer and a transform between hidden
        # layers, cropped by a box, a level other than zero, the mesh turned inside out
        {"name": "ragged_skip_mixed", "kind": "march", "net": 9, "widths": "100,72,130,45", "form": "mixed",
         "perturb": 0.01, "skip": "both", "box": 0.7, "level": 0.45, "flip": True, "seeds": 777},
        # the deep perturbed configuration at a level that closes
        {"name": "deep256x6_mixed", "kind": "march", "net": 2, "widths": "256,256,256,256,256,256", "form": "mixed",
         "perturb": 0.02, "level": 0.5, "seeds": 1024},
        # the largest single-network configuration: the input added into layer 4
        {"name": "skip512x8_mixed", "kind": "march", "net": 3, "widths": "512,512,512,512,512,512,512,512",
         "form": "mixed", "perturb": 0.01, "radius": 0.6, "skip": "input", "seeds": 1024},
        # the voxel mode's pattern: one network in the eight octants of a cube, six
        # extra constraints each, in the reference's default precision
        {"name": "octants64x3_f64", "kind": "batch", "net": 104, "nets": "64x3", "boxes": 8, "form": "float64",
         "perturb": 0.01, "seeds": 1024},
        # networks of the batched configuration's widths and depths, side by side
        {"name": "batch8_mixed", "kind": "batch", "net": 100, "nets": "32x2,64x4,128x3,32x8,256x2,64x6,128x5,256x3",
         "form": "mixed", "perturb": 0.01, "seeds": 1024},
        # constraint rows of activation states a program has in hand
        {"name": "rows128x4_8192", "kind": "rows", "net": 1, "widths": "128,128,128,128", "count": 8192},
    ]


def _widths(case):
    return [int(w) for w in case["widths"].split(",")]


def _regions(widths, perturb):
    n = sum(widths)
    return n * n * (DENSITY["perturbed"] if perturb else DENSITY["plain"])


def _capacity(widths, case):
    """Faces that a marching's arrays have room for."""
    r = _regions(widths, case.get("perturb", 0.0))
    return int(1.25 * r + 3.0 * min(r, 500000.0)) + 2048


def _flops(widths):
    """One region's composition: 4 columns, 2 flop per multiply-add."""
    return 8.0 * (sum(a * b for a, b in zip(widths, widths[1:])) + widths[-1])


def _seconds(form, widths, perturb):
    """A rough time of a marching, to keep drawn cases below the largest listed one."""
    rate = {"float64": 5e11, "float32": 1e13, "mixed": 1e14}[form]
    per_row = {"float64": 1.5e-9, "float32": 5e-11, "mixed": 5e-11}[form]
    return _regions(widths, perturb) * (_flops(widths) / rate + sum(widths) * per_row)


def draw(rng):
    kind = rng.choice(["march", "march", "march", "march", "batch", "rows"])
    net = rng.randint(1, 10000)
    if kind == "rows":
        depth = rng.randint(1, 6)
        widths = [int(round(2 ** rng.uniform(4, 8))) for _ in range(depth)]
        return {"kind": "rows", "net": net, "widths": ",".join(map(str, widths)),
                "count": int(round(2 ** rng.uniform(0, 13)))}
    form = rng.choice(["float32", "float64", "mixed", "mixed"])
    if kind == "batch":
        nets = []
        while len(nets) < rng.choice([2, 4, 8, 12]):
            w, d = int(round(2 ** rng.uniform(4, 8 if form == "mixed" else 6))), rng.randint(2, 6)
            if _seconds(form, [w] * d, 0.01) < 0.02 and w * d <= 700:
                nets.append("%dx%d" % (w, d))
        return {"kind": "batch", "net": net, "nets": ",".join(nets), "form": form, "perturb": 0.01,
                "seeds": rng.choice([256, 1024])}
    if form == "mixed" and rng.random() < 0.15:  # the large configurations from other seed points
        case = dict(rng.choice([c for c in listed() if c["name"] in ("deep256x6_mixed", "skip512x8_mixed")]))
        del case["name"]
        return {**case, "seeds": int(round(2 ** rng.uniform(6, 11)))}
    while True:
        depth = rng.randint(1, 8)
        width = 2 ** rng.uniform(4.5, 9)
        ragged = rng.random() < 0.5
        widths = [int(round(width * (rng.uniform(0.7, 1.3) if ragged else 1.0))) for _ in range(depth)]
        perturb = rng.choice([0.0, 0.01, 0.02])
        # plain float32 does not converge on the widest networks, and the mixed form
        # does not end on layers of 257 to 384 units
        if form == "mixed" and any(256 < w <= 384 or w > 512 for w in widths):
            continue
        most = 700 if form == "float32" else 3000
        if sum(widths) <= most and _seconds(form, widths, perturb) < 0.3:
            break
    case = {"kind": "march", "net": net, "widths": ",".join(map(str, widths)), "form": form, "perturb": perturb,
            "level": 0.5 if perturb or min(widths) < 64 else rng.choice([0.0, 0.5]),
            "seeds": int(round(2 ** rng.uniform(6, 11)))}
    if depth >= 3 and rng.random() < 0.4:
        case["skip"] = rng.choice(["input", "both"])
    if rng.random() < 0.25:
        case["box"] = 0.6
    return case


def _model(case, widths, net, seed):
    """A snapshot of the seeded network; "skip": the input added into the middle
    layer through a transform, for "both" hidden layer 1 into the last hidden one too."""
    if case.get("polytope"):
        return workloads.polytope(seed)
    n_lin = len(widths) + 1
    skips, shapes = None, None
    how = case.get("skip", "none")
    if how != "none" and len(widths) >= 3:
        skips = [[0, 0, 0, 0, 0] for _ in range(n_lin - 1)]
        mid = len(widths) // 2
        skips[mid - 1][:3] = [1, 0, 0]
        shapes = [[widths[mid], 3]]
        if how == "both":
            row = skips[len(widths) - 2]
            c = row[0]
            row[0] = c + 1
            row[1 + 2 * c:3 + 2 * c] = [1, 1]
            shapes.append([widths[-1], widths[0]])
    model = workloads.geometric(widths, net, radius=case.get("radius", 0.5), perturb=case.get("perturb", 0.0),
                                skips=skips, tm_shapes=shapes)
    g = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in model.parameters():
            p.mul_(1 + 1e-3 * torch.randn(p.shape, generator=g))
    return model


def _level(model, radius, seed):
    """The network's mean value on the sphere of that radius (0: level zero)."""
    if not radius:
        return 0.0
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(4096, 3, generator=g)
    x = radius * x / x.norm(dim=1, keepdim=True)
    with torch.no_grad():
        return float(model(x).double().mean())


def _on_device(net, form):
    """The network's arrays on the GPU in the form's own type."""
    tt = torch.float64 if form == "float64" else torch.float32
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to("cuda", tt).contiguous()
    return workloads.NetArrays(nodes=net.nodes, W=[f(w) for w in net.W], b=[f(b) for b in net.b],
                               arc_table=net.arc_table, tms=[f(t) for t in net.tms], w_extra=f(net.w_extra),
                               b_extra=f(net.b_extra)), tt


def _box(lo, hi):
    return utils.get_boundary("cube", min_vert=lo, max_vert=hi)


def _states(model, points):
    """Activation states of given points, from a float64 forward pass on the GPU."""
    m = workloads._double_copy(model).to("cuda")
    with torch.no_grad():
        return (m.pre_activations(points.double()) > 0).to(torch.uint8).contiguous()


def _network(case, widths, net, seed, box=None):
    """One network as a program holds it before the call: (arrays, seed states, seed points, level)."""
    model = _model(case, widths, net, seed)
    iso = _level(model, case.get("level", 0.0), seed + 1)
    we = be = None
    if box is not None:
        we, be = _box(*box)
    states, points = workloads.seeds_for(model, init_num=case["seeds"], seed=seed + 2, iso=iso, w_extra=we,
                                         b_extra=be, device="cuda")
    host = workloads.net_arrays(model, we, be)
    net, tt = _on_device(host, case["form"])
    return {"net": net, "host": host, "states": torch.as_tensor(states).cuda(),
            "points": torch.as_tensor(points).to("cuda", tt), "iso": iso}


def _case_networks(case, seed):
    if case["kind"] == "march":
        b = case.get("box", 0.0)
        return [_network(case, _widths(case), case.get("net", 0), seed, ([-b] * 3, [b] * 3) if b else None)]
    shapes = [[int(w)] * int(d) for w, d in (s.split("x") for s in case["nets"].split(","))]
    if case.get("boxes"):  # the octants of [-0.7, 0.7]^3, as occupied voxels
        out = []
        for o in range(case["boxes"]):
            lo = [-0.7 if (o >> a) & 1 else 0.0 for a in range(3)]
            out.append(_network(case, shapes[0], case["net"], seed, (lo, [x + 0.7 for x in lo])))
        return out
    return [_network(case, w, case["net"] + i, seed + 10 * i) for i, w in enumerate(shapes)]


def prepare(case, seed):
    seed = 1000 + seed % 1000003
    if case["kind"] == "rows":
        widths = _widths(case)
        model = _model(case, widths, case["net"], seed)
        g = torch.Generator().manual_seed(seed)
        pts = torch.rand(case["count"], 3, generator=g) * 2 - 1
        states = _states(model, pts.cuda())
        net, _ = _on_device(workloads.net_arrays(model), "float32")
        n = sum(widths)
        return {"kind": "rows", "net": net, "states": states,
                "rows": torch.zeros(case["count"], n, 4, device="cuda"),
                "eq": torch.zeros(case["count"], 4, device="cuda")}
    items = _case_networks(case, seed)
    for it in items:
        it["engine"] = engine.Engine(case["form"], it["net"].nodes, it["net"].arc_table, it["net"].num_extra)
        faces = _capacity(it["net"].nodes[1:-1], case)
        it["verts"] = np.zeros((faces * 3 // 2, 3))
        it["face_sizes"] = np.zeros(faces, np.int32)
        it["face_indices"] = np.zeros(6 * faces, np.int32)
    return {"kind": case["kind"], "items": items, "flip": bool(case.get("flip", False))}


def _mesh(it):
    """The welded mesh of the engine's last run into the program's arrays."""
    L, h = _lib.lib(), it["engine"].h
    _lib.check(L.am_combine_mesh(h, 1.0, (ctypes.c_double * 3)(0.0, 0.0, 0.0)), h)
    s = it["engine"].stats()
    if (s["mesh_num_verts"] > len(it["verts"]) or s["mesh_num_faces"] > len(it["face_sizes"]) or
            s["mesh_num_indices"] > len(it["face_indices"])):
        raise RuntimeError("a mesh of %d faces does not fit" % s["mesh_num_faces"])
    _lib.check(L.am_get_mesh(h, it["verts"].ctypes.data, it["face_sizes"].ctypes.data,
                             it["face_indices"].ctypes.data), h)
    return {"verts": it["verts"], "face_sizes": it["face_sizes"], "face_indices": it["face_indices"]}


def run(state):
    if state["kind"] == "rows":
        net = state["net"]
        nodes = (ctypes.c_int32 * len(net.nodes))(*net.nodes)
        ws = (ctypes.c_void_p * len(net.W))(*[w.data_ptr() for w in net.W])
        bs = (ctypes.c_void_p * len(net.b))(*[b.data_ptr() for b in net.b])
        _lib.check(_lib.lib().am_compose_rows_noalloc(
            nodes, len(net.nodes), ws, bs, state["states"].data_ptr(), int(state["states"].shape[0]), 0.0,
            state["rows"].data_ptr(), state["eq"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return {"rows": state["rows"], "eq": state["eq"]}
    items = state["items"]
    if state["kind"] == "march":
        it = items[0]
        stats = it["engine"].run_net(it["net"], it["states"], it["points"], it["iso"], state["flip"])
        return {**_mesh(it), "regions": stats["num_regions"], "faces": stats["num_faces"]}
    engine.run_batch([it["engine"] for it in items], [it["net"] for it in items], [it["states"] for it in items],
                     [it["points"] for it in items], items[0]["iso"], state["flip"])
    return [_mesh(it) for it in items]


def work(case):
    """Bytes: the parameters and seeds read, the mesh (or the rows) written.
    Flops: half of every region's layer products -- a region shares the layers
    before the plane it was entered through with its neighbour -- and one
    signed distance per region and constraint."""
    size = 8 if case.get("form") == "float64" else 4
    if case["kind"] == "rows":
        widths, n = _widths(case), sum(_widths(case))
        params = sum(a * b + b for a, b in zip([3] + widths, widths + [1]))
        return {"bytes": 4.0 * params + case["count"] * (n + 16.0 * n + 16), "flops": case["count"] * _flops(widths)}
    if case["kind"] == "march":
        shapes = [_widths(case)]
    else:
        shapes = [[int(w)] * int(d) for w, d in (s.split("x") for s in case["nets"].split(","))]
    total = {"bytes": 0.0, "flops": 0.0}
    for widths in shapes:
        n, regions = sum(widths), _regions(widths, case.get("perturb", 0.0))
        if case.get("polytope"):  # a closed convex surface of tens of faces
            regions = 60.0
        params = sum(a * b + b for a, b in zip([3] + widths, widths + [1]))
        total["bytes"] += size * params + case["seeds"] * (n + 3.0 * size) + regions * (24 + 4 + 16)
        total["flops"] += regions * (0.5 * _flops(widths) + 8.0 * n)
    return total


# ------------------------------------------------------------------ exact
def _exact_rows(net, states):
    """Rows and face planes of given states in float64: C = (1 - 2 s) A."""
    W = [w.double() for w in net.W]
    b = [x.double() for x in net.b]
    s = states.double()
    A = torch.cat([W[0], b[0][:, None]], dim=1).expand(s.shape[0], -1, -1)
    rows, o = [], 0
    for i in range(1, len(W)):
        n = W[i - 1].shape[0]
        sl = s[:, o:o + n, None]
        rows.append((1 - 2 * sl) * A)
        A = torch.matmul(W[i], sl * A)
        A[:, :, 3] += b[i]
        o += n
    return torch.cat(rows, dim=1), A[:, 0, :]


def _solve(r0, r1, r2):
    m = np.array([r0[:3], r1[:3], r2[:3]])
    rhs = -np.array([r0[3], r1[3], r2[3]])
    d = np.linalg.det(m)
    out = np.empty(3)
    for c in range(3):
        t = m.copy()
        t[:, c] = rhs
        out[c] = np.linalg.det(t) / d if d else np.inf
    return out


def _pair(x, most):
    k = x // 2
    a = int(math.ceil(math.sqrt(2 * k + 2.25) - 1.5))
    r = x - a * (a + 1)
    s, t = 2 * a + r // (a + 1), r % (a + 1)
    i = (s + 1) // 2 + t + 1
    return min(i, most - 1), min(s + 1 - i, most - 1)


def _exact_march(net, states, points, iso, same):
    """Analytic Marching of a plain network in float64 numpy: regions first in,
    first out, each face walked around its plane; the welded mesh."""
    W, B = [w.double().cpu().numpy() for w in net.W], [b.double().cpu().numpy() for b in net.b]
    offs = np.cumsum([0] + [w.shape[0] for w in W[:-1]])
    seen, queue = {}, []
    for st, pt in zip(states.cpu().numpy().astype(bool), points.double().cpu().numpy()):
        if st.tobytes() not in seen:
            seen[st.tobytes()] = len(queue)
            queue.append((st, pt, -1))
    weld, verts, sizes, index = {}, [], [], []
    q = 0
    while q < len(queue):
        key, p, s = queue[q]
        q += 1
        A = np.concatenate([W[0], B[0][:, None]], axis=1)
        rows = []
        for i in range(1, len(W)):
            act = key[offs[i - 1]:offs[i]]
            rows.append(np.where(act[:, None], -A, A))
            A = W[i] @ (A * act[:, None])
            A[:, 3] += B[i]
        eq = A[0].copy()
        eq[3] -= iso
        R = np.concatenate(rows)
        norm = np.linalg.norm(R[:, :3], axis=1)
        R = R / np.where(norm > 0, norm, 1.0)[:, None]
        R[norm == 0, 3] = np.where(R[norm == 0, 3] > 0, np.inf, -np.inf)
        seed = s < 0
        if seed:
            order = np.argsort(-(R[:, :3] @ p + R[:, 3]), kind="stable")
            most = len(order)
            for x in range(min((most - 1) * (most - 2), 812) + 1):
                i, j = _pair(x, most)
                v = _solve(R[order[i]], R[order[j]], eq)
                g = R[:, :3] @ v + R[:, 3]
                g[[order[i], order[j]]] = -1
                if np.all(g <= 1e-12):
                    s, p = int(order[i]), v
                    break
            if s < 0:
                continue
        V, E, e, prev, cur, closed = [], [], s, -1, p, False
        for _ in range(96):
            d = np.cross(eq[:3], R[e, :3])
            a = R[:, :3] @ d
            ok = a > 1e-12 * np.linalg.norm(d)
            ok[e] = False
            if prev >= 0:
                ok[prev] = False
            if not ok.any():
                break
            t = np.full(len(a), np.inf)
            t[ok] = np.maximum(0.0, -(R[ok, :3] @ cur + R[ok, 3])) / a[ok]
            hit = int(np.argmin(t))
            v = _solve(R[e], R[hit], eq)
            if V and np.abs(v - V[-1]).sum() < same:
                E[-1] = hit
            elif not (V and hit == s and np.abs(v - V[0]).sum() < same):
                V.append(v)
                E.append(hit)
            if hit == s:
                closed = True
                break
            if len(V) >= 32:
                break
            prev, e, cur = e, hit, v
        n = len(V)
        for i in range(n):
            k = E[i]
            if not (closed or i < n - 1) or (not seed and k == s):
                continue
            child = key.copy()
            child[k] ^= True
            if child.tobytes() not in seen:
                seen[child.tobytes()] = len(queue)
                queue.append((child, (V[i] + V[(i + 1) % n]) / 2, k))
        ids = []
        for i in range(n):
            pq = sorted((E[i - 1], E[i]))
            bits = key.copy()
            bits[pq] = False
            name = (pq[0], pq[1], bits.tobytes())
            if name not in weld:
                weld[name] = len(verts)
                verts.append(V[i])
            ids.append(weld[name])
        if n >= 3:
            sizes.append(n)
            index += ids
    return {"verts": np.array(verts).reshape(-1, 3), "face_sizes": np.array(sizes, np.int32),
            "face_indices": np.array(index, np.int32), "regions": len(queue), "faces": len(sizes)}


def exact(case, seed):
    if case["kind"] == "rows":
        state = prepare(case, seed)
        rows, eq = [], []
        for st in state["states"].split(1024):
            r, e = _exact_rows(state["net"], st)
            rows.append(r)
            eq.append(e)
        return {"rows": torch.cat(rows), "eq": torch.cat(eq)}
    # a marching of more regions takes this plain program too long
    if (case["kind"] != "march" or case.get("skip") or case.get("box") or case.get("flip") or
            _regions(_widths(case), case.get("perturb", 0.0)) > 6000):
        return None
    it = _case_networks(case, 1000 + seed % 1000003)[0]
    out = _exact_march(it["net"], it["states"], it["points"], it["iso"], 3e-14 if case["form"] == "float64" else 3e-7)
    faces = _capacity(_widths(case), case)
    for name, room in (("verts", faces * 3 // 2), ("face_sizes", faces), ("face_indices", 6 * faces)):
        full = np.zeros((room,) + out[name].shape[1:], out[name].dtype)
        full[:len(out[name])] = out[name]
        out[name] = full
    return out
