"""What the framework is timed on: its public Python entry points over the
sizes, types and options of the benchmark configurations, of the tests and of
generic scientific fields (2^k + 1 grids, even and ragged ones).

listed() gives the fixed cases, draw(rng) further ones of the same ranges,
prepare(case, seed) what a program has in hand before the call, run(state) one
pass, work(case) the bytes and operations a pass cannot do without and
exact(case, seed) the same outputs from 64-bit arithmetic without this
package, where they have such a value.

A retrieval approximates the field that was refactored, so the 64-bit value of
a retrieved field is that field: the error of a pass is the error a reader of
the data sees, the planes left out included. Streams and metadata are bytes
and have no such value.
"""
import math

import numpy as np
import torch

DTYPES = {"f32": torch.float32, "f64": torch.float64}


# ---------------------------------------------------------------------------
# geometry
# ---------------------------------------------------------------------------
def shape_of(case):
    return tuple(int(n) for n in case["shape"].split("x"))


def size_of(case):
    return math.prod(shape_of(case))


def levels_of(shape, block):
    """Target level: as deep as the smallest dim allows, at most 9, with one
    full block of values left at level 0."""
    most = min(9, int(math.log2(min(shape)) - 1))
    for level in range(most, 0, -1):
        box = shape
        for _ in range(level):
            box = tuple((n >> 1) + 1 for n in box)
        if math.prod(box) >= block:
            return level
    return 0


def block_of(case):
    return 64 if case.get("dtype") == "f64" else 32


def boxes_of(shape, level):
    """Boxes of levels 0 .. level."""
    boxes = [tuple(shape)]
    for _ in range(level):
        boxes.insert(0, tuple((n >> 1) + 1 for n in boxes[0]))
    return boxes


# ---------------------------------------------------------------------------
# inputs, each from its seed alone
# ---------------------------------------------------------------------------
def generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def spectral_field(shape, seed, slope=-5.0 / 3.0):
    """Gaussian random field with power spectrum k^slope and unit variance, fp32."""
    white = torch.randn(shape, dtype=torch.float32, device="cuda", generator=generator(seed))
    spec = torch.fft.rfftn(white)
    kk = torch.zeros((), device="cuda")
    for i, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device="cuda") if i == len(shape) - 1 else torch.fft.fftfreq(n, device="cuda")
        view = [1] * len(shape)
        view[i] = -1
        kk = kk + ((k * n) ** 2).view(view)
    kk.view(-1)[0] = 1.0
    amp = kk.pow_(slope / 4.0)
    amp.view(-1)[0] = 0.0
    f = torch.fft.irfftn(spec.mul_(amp), s=shape)
    return (f / f.std()).contiguous()


def wave_field(shape, seed):
    """Four sinusoids of random phase (wavenumbers 1 to 8) plus noise, fp32."""
    rng = np.random.default_rng(seed)
    f = 1e-3 * torch.randn(shape, dtype=torch.float32, device="cuda", generator=generator(seed))
    for _ in range(4):
        arg = torch.zeros((), device="cuda")
        for i, n in enumerate(shape):
            view = [1] * len(shape)
            view[i] = -1
            k = float(rng.integers(1, 9) * rng.choice([-1, 1]))
            arg = arg + (2 * math.pi * k / n) * torch.arange(n, device="cuda").view(view)
        f += torch.sin(arg + float(rng.uniform(0, 2 * math.pi)))
    return f.contiguous()


def shear_field(shape, seed):
    """tanh shear layer across one dim plus 1e-6 relative white noise, fp64."""
    dim = max(0, len(shape) - 2)
    view = [1] * len(shape)
    view[dim] = -1
    prof = torch.tanh((torch.linspace(0.0, 1.0, shape[dim], dtype=torch.float64, device="cuda") - 0.5) / 0.05)
    noise = torch.randn(shape, dtype=torch.float64, device="cuda", generator=generator(seed))
    return noise.mul_(2e-6).add_(prof.view(view)).contiguous()


def field_of(case, seed):
    shape = shape_of(case)
    if case["field"] == "spectral":
        return spectral_field(shape, seed).to(DTYPES[case["dtype"]])
    if case["field"] == "waves":
        return wave_field(shape, seed).to(DTYPES[case["dtype"]])
    return shear_field(shape, seed).to(DTYPES[case["dtype"]])


def rels_of(case):
    return [float(r) for r in case["rels"].split(",")]


def batch_of(case):
    """(shape, spectral slope, relative tolerance) of every field of a batch:
    of the benchmark's families (cubes, planes, anisotropic boxes), or of free
    sizes up to the same ones."""
    rng = np.random.default_rng(case["spec"])
    specs = []
    for i in range(case["fields"]):
        if case["family"] == "grid":
            part = i * 64 // case["fields"]
            if part < 24:
                shape = (int(rng.choice([33, 65, 129, 257])),) * 3
            elif part < 48:
                shape = (int(rng.choice([513, 1025, 2049])),) * 2
            else:
                shape = (129, 257, 65)
        elif rng.uniform() < 0.6:
            shape = tuple(int(n) for n in np.exp(rng.uniform(math.log(24), math.log(200), 3)))
        else:
            shape = tuple(int(n) for n in np.exp(rng.uniform(math.log(100), math.log(1500), 2)))
        specs.append((shape, float(rng.uniform(-3.0, -1.0)), float(10.0 ** rng.uniform(-5.0, -2.0))))
    return specs


def flow_of(case, seed):
    """Velocity components, pressure (around 1 bar) and density of n points, fp64."""
    n = case["points"]
    g = generator(seed)
    v = [30.0 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g) for _ in range(3)]
    rho = torch.exp(0.5 * torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    p = 1e5 * (1.0 + 0.1 * rho)
    return v[0], v[1], v[2], p, rho


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # A small field through the whole path, as in a time loop that keeps many small blocks: grouped encoder, five
        # progressive tolerances (the 65^3 configuration of the benchmark). Launches and latency count.
        {"name": "small_cube_grouped", "kind": "step", "shape": "65x65x65", "dtype": "f32", "field": "waves",
         "encoder": "grouped", "basis": "hierarchical", "rels": "3e-2,1e-2,1e-3,1e-4,1e-5"},
        # The headline field, written with squared-error tables and read at five progressive L2 tolerances.
        {"name": "large_cube", "kind": "step", "shape": "513x513x513", "dtype": "f32", "field": "spectral",
         "encoder": "negabinary", "basis": "hierarchical", "collector": "squared", "rels": "1e-2,1e-3,1e-4,1e-5,1e-6"},
        # A simulation's slab with even sizes (no 2^k + 1 dim), written and read at three tolerances.
        {"name": "even_slab", "kind": "step", "shape": "100x500x500", "dtype": "f32", "field": "spectral",
         "encoder": "negabinary", "basis": "hierarchical", "rels": "1e-2,1e-3,1e-4"},
        # A 2-D map with even sizes, as climate fields have.
        {"name": "even_plane", "kind": "step", "shape": "1800x3600", "dtype": "f32", "field": "spectral",
         "encoder": "negabinary", "basis": "hierarchical", "rels": "1e-2,1e-3,1e-4"},
        # Double precision with the L2-projected basis (a part of the 1025 x 1025 x 513 configuration).
        {"name": "f64_orthogonal", "kind": "step", "shape": "513x513x257", "dtype": "f64", "field": "shear",
         "encoder": "grouped", "basis": "orthogonal", "rels": "1e-3,1e-6,1e-9"},
        # The GE applications' encoder on resident data: fp64, per-bit, 60 planes.
        {"name": "f64_perbit", "kind": "step", "shape": "513x257x257", "dtype": "f64", "field": "shear",
         "encoder": "perbit", "basis": "hierarchical", "rels": "1e-3,1e-5,1e-7,1e-9"},
        # The GE applications' files: per-bit level files through the lossless stage, written, read back and retrieved.
        {"name": "perbit_files", "kind": "files", "shape": "129x129x129", "dtype": "f64", "field": "shear",
         "encoder": "perbit", "basis": "hierarchical", "lossless": True, "rels": "1e-7"},
        # Level files of a simulation block through the lossless stage, written, read back and retrieved.
        {"name": "lossless_files", "kind": "files", "shape": "257x257x257", "dtype": "f32", "field": "spectral",
         "encoder": "negabinary", "basis": "hierarchical", "lossless": True, "rels": "1e-4"},
        # Many fields of uneven sizes at once: the 64-field batch.
        {"name": "batch64", "kind": "batch", "fields": 64, "family": "grid", "spec": 7},
        # GE quantities of interest and their error estimates on a retrieved flow.
        {"name": "qoi_flow", "kind": "qoi", "points": 257 * 257 * 257},
        # Forward and adjoint recomposition of packed coefficients (QoI-bounded retrieval).
        {"name": "packed_adjoint", "kind": "adjoint", "shape": "257x257x257", "dtype": "f32", "field": "spectral",
         "basis": "hierarchical"},
        # The reference's composition out of single components (decomposer, interleaver, encoder and back), ragged sizes.
        {"name": "components", "kind": "components", "shape": "150x257x301", "dtype": "f32", "field": "spectral",
         "encoder": "grouped", "basis": "hierarchical"},
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "refactor", "retrieve", "batch", "files", "qoi", "adjoint", "components"])
    if kind == "qoi":
        return {"kind": kind, "points": int(math.exp(rng.uniform(math.log(1 << 12), math.log(1 << 24))))}
    if kind == "batch":
        return {"kind": kind, "fields": rng.randint(4, 64), "family": rng.choice(["grid", "free"]),
                "spec": rng.randrange(1 << 20)}
    dtype = rng.choice(["f32", "f32", "f64"])
    encoder = rng.choice(["negabinary", "grouped"] if dtype == "f32" else ["grouped", "perbit", "negabinary"])
    basis = rng.choice(["hierarchical", "hierarchical", "hierarchical", "orthogonal"])
    most = {"refactor": 27, "retrieve": 27, "step": 26, "files": 24, "adjoint": 24.5, "components": 23.5}[kind]
    if dtype == "f64":
        most = min(most, 25)
    if basis == "orthogonal":
        most = min(most, 24)
    if encoder == "perbit" and kind in ("files", "components"):
        most = min(most, 20)
    total = 2.0 ** rng.uniform(14, most)
    ndims = rng.choice([1, 2, 2, 3, 3, 3, 3])
    if ndims == 1:
        total = min(total, 2.0 ** 24)
    part = [math.exp(rng.uniform(-0.6, 0.6)) for _ in range(ndims)]
    scale = (total / math.prod(part)) ** (1.0 / ndims)
    shape = [max(8, int(scale * f)) for f in part]
    if ndims > 1 and rng.random() < 0.35:   # a 2^k + 1 grid near the same size
        shape = [(1 << max(3, int(math.log2(n)))) + 1 for n in shape]
    case = {"kind": kind, "shape": "x".join(str(n) for n in shape), "dtype": dtype,
            "field": "shear" if dtype == "f64" else rng.choice(["spectral", "waves"]), "basis": basis}
    if kind != "adjoint":
        case["encoder"] = encoder
    if kind in ("step", "refactor", "retrieve") and basis == "hierarchical" and dtype == "f32":
        case["collector"] = rng.choice(["max", "squared"])
    if kind == "files":
        case["lossless"] = rng.random() < 0.6
    if kind in ("step", "retrieve", "files"):
        lo, hi = (-4, -2) if dtype == "f32" else (-8, -2)
        count = 1 if kind == "files" else rng.randint(1, 4)
        exps = sorted((round(rng.uniform(lo, hi), 2) for _ in range(count)), reverse=True)
        case["rels"] = ",".join("%.3e" % 10.0 ** e for e in exps)
    return case


def planes_of(case):
    return 32 if case.get("dtype", "f32") == "f32" else 60


def stored_bound(case):
    """Bytes that the level files of a field take at most, each from a 64-byte boundary on."""
    shape, block, planes = shape_of(case), block_of(case), planes_of(case)
    boxes = boxes_of(shape, levels_of(shape, block))
    total = 0
    for i, box in enumerate(boxes):
        blocks = -(-(math.prod(box) - (math.prod(boxes[i - 1]) if i else 0)) // block)
        total += blocks * ((planes + 1) * block // 8 + 1) + 32 * planes + 68
    return total


def handle_of(case):
    from prodm_gb300 import api
    shape = shape_of(case)
    return api.MDRField(shape, DTYPES[case["dtype"]], levels_of(shape, block_of(case)), planes_of(case), case["encoder"],
                        case["basis"], case.get("collector", "max"))


def options_of(case):
    """Interpreter and estimator of a retrieval, as the reference pairs them."""
    interpreter = "negabinary" if case["encoder"] == "negabinary" else "sign_exclude"
    if case.get("collector") == "squared":
        return {"interpreter": interpreter, "estimator": "l2_hb"}
    return {"interpreter": interpreter, "estimator": "max_hb" if case["basis"] == "hierarchical" else "max_ob"}


def tolerances_of(case, x):
    """Absolute tolerances: of the squared L2 norm, or of the value range."""
    if case.get("collector") == "squared":
        norm2 = float((x.double() ** 2).sum())
        return [r * r * norm2 for r in rels_of(case)]
    span = float(x.max() - x.min())
    return [r * span for r in rels_of(case)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "qoi":
        return {"kind": kind, "flow": flow_of(case, seed)}
    if kind == "batch":
        from prodm_gb300 import api
        xs, tols, levels = [], [], []
        for i, (shape, slope, rel) in enumerate(batch_of(case)):
            xs.append(spectral_field(shape, 1000 * seed + i, slope))
            tols.append(rel * (xs[-1].max() - xs[-1].min()))
            levels.append(levels_of(shape, 32))
        batch = api.MDRBatch(xs, levels, 32)
        batch.set_tolerances(torch.stack(tols).tolist())
        return {"kind": kind, "batch": batch}
    if kind == "adjoint":
        return packed_of(case, seed)
    x = field_of(case, seed)
    state = {"kind": kind, "x": x, "shape": shape_of(case), "level": levels_of(shape_of(case), block_of(case)),
             "basis": case["basis"]}
    if kind == "components":
        state.update(encoder=case["encoder"], planes=planes_of(case), boxes=boxes_of(state["shape"], state["level"]),
                     image=torch.zeros(stored_bound(case), dtype=torch.uint8, device="cuda"))
        return state
    state["m"] = handle_of(case)
    if "rels" in case:
        state["tols"], state["options"] = tolerances_of(case, x), options_of(case)
        state["outs"] = [torch.empty_like(x) for _ in state["tols"]]
    if kind == "retrieve":
        state["m"].refactor(x)
    if kind in ("refactor", "files"):
        # one buffer for all level files; the lossless stage may store a few bytes more than the plane's own
        state["image"] = torch.zeros(stored_bound(case) * 9 // 8 + (1 << 16), dtype=torch.uint8, device="cuda")
    if kind == "files":
        if case["lossless"]:
            state["m"].set_lossless(26)
        state["reader"] = handle_of(case)
    return state


def retrieve(m, state):
    m.reset()
    for tol, out in zip(state["tols"], state["outs"]):
        m.retrieve(tol, out=out, **state["options"])
    return state["outs"]


def level_files(m, level, image):
    """The level files, one after the other in `image` (each from a 64-byte
    boundary on), their places, and the metadata, as a writer takes them."""
    at, places = 0, []
    for i in range(level + 1):
        n = m.export_level_into(i, image[at:])
        places.append((at, n))
        at = (at + n + 63) // 64 * 64
    return places, np.frombuffer(m.metadata(), np.uint8)


def components(state):
    """ComposedRefactor's and ComposedReconstructor's loops out of the single components."""
    from prodm_gb300 import api
    x, level, boxes, kind, planes = state["x"], state["level"], state["boxes"], state["encoder"], state["planes"]
    data = api.decompose(x.clone(), level, basis=state["basis"])
    rec = torch.empty_like(x)
    decoder = api.ProgressiveDecoder(kind, x.dtype)
    at = 0
    for i, box in enumerate(boxes):
        coarse = boxes[i - 1] if i else (0,) * len(box)
        coef = api.interleave(data, box, coarse)
        exp = math.frexp(float(coef.abs().max()))[1]
        blob, sizes, _ = api.encode(kind, coef, exp, planes)
        state["image"][at:at + blob.numel()].copy_(blob)
        at = (at + blob.numel() + 63) // 64 * 64
        back = decoder.decode(blob, sizes, coef.numel(), exp, 0, planes, i, planes)
        api.reposition(back, rec, box, coarse)
    return data, state["image"], api.recompose(rec, level, basis=state["basis"])


def run(state):
    from prodm_gb300 import api
    kind = state["kind"]
    if kind == "step":
        state["m"].refactor(state["x"])
        return retrieve(state["m"], state)
    if kind == "refactor":
        state["m"].refactor(state["x"])
        places, meta = level_files(state["m"], state["level"], state["image"])
        return state["image"], np.array(places), meta
    if kind == "retrieve":
        return retrieve(state["m"], state)
    if kind == "batch":
        state["batch"].refactor()
        state["batch"].reset()
        return state["batch"].retrieve("negabinary", "max_hb")
    if kind == "files":
        state["m"].refactor(state["x"])
        places, meta = level_files(state["m"], state["level"], state["image"])
        state["reader"].load_metadata(meta.tobytes())
        for i, (at, n) in enumerate(places):
            state["reader"].load_level(i, state["image"][at:at + n])
        return state["image"], np.array(places), meta, retrieve(state["reader"], state)
    if kind == "qoi":
        vx, vy, vz, p, d = state["flow"]
        return api.qoi_ge_values(vx, vy, vz, p, d), api.qoi_ge_bounds([vx, vy, vz], (0.01, 0.01, 0.01), p, d, 10.0, 1e-4)
    if kind == "adjoint":
        return (api.recompose_packed(state["coef"], state["shape"], state["level"], basis=state["basis"]),
                api.recompose_adjoint(state["grad"], state["level"], basis=state["basis"]))
    return components(state)


def work(case):
    """A refactor reads the field and writes every plane; a retrieval reads about
    log2(1 / tolerance) + 4 planes of the values and writes the field. Per value
    and direction the transform adds or subtracts about three times."""
    kind = case["kind"]
    if kind == "qoi":
        return {"bytes": 8 * case["points"] * (5 + 6 + 5 + 2), "flops": 50 * case["points"]}

    def planes_read(rel):
        return min(planes_of(case), math.log2(1.0 / rel) + 4)

    if kind == "batch":
        total = sum(math.prod(s) * (4 + 4 + planes_read(r) / 8 + 4) for s, _, r in batch_of(case))
        return {"bytes": total, "flops": 6 * sum(math.prod(s) for s, _, _ in batch_of(case))}
    n, es, stored = size_of(case), 4 if case["dtype"] == "f32" else 8, planes_of(case) / 8
    read = sum(n * (es + planes_read(r) / 8) for r in rels_of(case)) if "rels" in case else 0
    passes = len(rels_of(case)) if "rels" in case else 0
    write = n * (es + stored)
    if kind == "step":
        return {"bytes": write + read, "flops": 3 * n * (1 + passes)}
    if kind == "refactor":
        return {"bytes": write, "flops": 3 * n}
    if kind == "retrieve":
        return {"bytes": read, "flops": 3 * n * passes}
    if kind == "files":
        return {"bytes": write + n * stored + read, "flops": 6 * n}
    if kind == "adjoint":
        return {"bytes": 4 * n * es, "flops": 8 * n}
    return {"bytes": 2 * write, "flops": 6 * n}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def coarse_nodes(n):
    """Coarse nodes of one dim: the even ones below n - 1, and n - 1."""
    return list(range(0, n - 1, 2)) + [n - 1]


def odd_nodes(n):
    return list(range(1, n - 1, 2))


def interpolate(c, shape):
    """Multilinear interpolant on the fine grid of the coarse nodal values c."""
    for dim, n in enumerate(shape):
        even = torch.tensor(coarse_nodes(n), device=c.device)
        odd = torch.tensor(odd_nodes(n), device=c.device, dtype=torch.long)
        size = list(c.shape)
        size[dim] = n
        f = torch.zeros(size, dtype=c.dtype, device=c.device).index_copy(dim, even, c)
        left = c.index_select(dim, odd // 2)
        right = c.index_select(dim, odd // 2 + 1)
        c = f.index_copy(dim, odd, 0.5 * (left + right))
    return c


def reordered(f):
    """Coarse nodes first along every dim."""
    for dim, n in enumerate(f.shape):
        f = f.index_select(dim, torch.tensor(coarse_nodes(n) + odd_nodes(n), device=f.device))
    return f


def natural(f):
    for dim, n in enumerate(f.shape):
        order = torch.tensor(coarse_nodes(n) + odd_nodes(n), device=f.device)
        f = f.index_select(dim, torch.argsort(order))
    return f


def corner(box):
    return tuple(slice(0, n) for n in box)


def level_mask(box, coarse):
    mask = torch.ones(box, dtype=torch.bool, device="cuda")
    mask[corner(coarse)] = False
    return mask


def decomposed(x, boxes):
    """In-place layout of the hierarchical decomposition."""
    u = x.clone()
    for box, coarse in zip(boxes[:0:-1], boxes[-2::-1]):
        f = reordered(u[corner(box)])
        c = f[corner(coarse)].clone()
        f = f - reordered(interpolate(c, box))
        f[corner(coarse)] = c
        u[corner(box)] = f
    return u


def recomposed_packed(coef, boxes):
    """Natural-order field of packed level coefficients, hierarchical basis."""
    at = math.prod(boxes[0])
    u = coef[:at].view(boxes[0])
    for coarse, box in zip(boxes, boxes[1:]):
        mask = level_mask(box, coarse)
        n = math.prod(box) - math.prod(coarse)
        f = torch.zeros(box, dtype=coef.dtype, device=coef.device).masked_scatter(mask, coef[at:at + n])
        at += n
        u = interpolate(u, box) + natural(f)
    return u


def packed_of(case, seed):
    """Packed level coefficients of a field, and the gradient of a quantity of
    interest with respect to the recomposed field."""
    x = field_of(case, seed)
    shape = shape_of(case)
    level = levels_of(shape, block_of(case))
    boxes = boxes_of(shape, level)
    u = decomposed(x, boxes)
    coef = [u[corner(boxes[0])].reshape(-1)]
    for coarse, box in zip(boxes, boxes[1:]):
        coef.append(u[corner(box)][level_mask(box, coarse)])
    grad = torch.randn(shape, dtype=x.dtype, device="cuda", generator=generator(seed + 1))
    return {"kind": case["kind"], "coef": torch.cat(coef), "grad": grad, "shape": shape, "level": level,
            "basis": case["basis"]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "qoi":
        vx, vy, vz, p, d = flow_of(case, seed)
        gas, gamma = 287.1, 1.4
        v2 = vx * vx + vy * vy + vz * vz
        v = v2.sqrt()
        t = p / (d * gas)
        c = (gamma * gas * t).sqrt()
        mach = v / c
        pt = p * (1 + 0.5 * (gamma - 1) * mach * mach).pow(3.5)
        mu = 1.716e-5 * (t / 273.15).pow(1.5) * (273.15 + 110.4) / (t + 110.4)
        e2 = sum(2 * f.abs() * 0.01 + 0.01 * 0.01 for f in (vx, vy, vz))
        bv = torch.where(v2 > e2, e2 / ((v2 - e2).clamp_min(0).sqrt() + v), e2 / v)
        e, far = p * 1e-4 + d * 10.0, d > 1e-4
        bt = torch.where(far, e / (d * (d - 1e-4)), torch.zeros_like(e)) / gas
        return [v, t, c, mach, pt, mu], (bv, bt, torch.stack([bv.max(), bt.max()]))
    if kind == "batch":
        return [spectral_field(shape, 1000 * seed + i, slope).double()
                for i, (shape, slope, _) in enumerate(batch_of(case))]
    if kind == "refactor":
        return None
    if kind == "adjoint":
        if case["basis"] != "hierarchical":
            return None
        state = packed_of(case, seed)
        boxes = boxes_of(state["shape"], state["level"])
        with torch.enable_grad():
            coef = state["coef"].double().requires_grad_()
            out = recomposed_packed(coef, boxes)
            grad, = torch.autograd.grad(out, coef, state["grad"].double())
        return out.detach(), grad
    x = field_of(case, seed).double()
    if kind == "components":
        boxes = boxes_of(shape_of(case), levels_of(shape_of(case), block_of(case)))
        data = decomposed(x, boxes) if case["basis"] == "hierarchical" else None
        return data, None, x
    outs = [x for _ in rels_of(case)]
    return (None, None, None, outs) if kind == "files" else outs
