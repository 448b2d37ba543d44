"""The work that programs built on this library have it do, as measurable cases.

Every case is one pass of a program's main path through the public entry
points: a simulation run (cells in, time steps, cells out), calls of the
learned surrogate, or one training iteration.  Fields go in and out through
pinned host buffers where a program's Initializer and Writers hold them
(structured grids, SELL-C-sigma, ensembles) and stay in torch CUDA tensors
where the device pipeline does (plain stencil of the surrogate, network).

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, grids, matrices and networks
    run(state)           one pass, returns its outputs
    work(case)           bytes and flops one pass cannot do without
    exact(case, seed)    what run returns, in 64 bits, by torch alone
"""
import ctypes
import math

import numpy as np
import torch

from libgeodecomp_gb300 import lgd, surrogate

CHUNK, SIGMA = 32, 256          # SELL-C-sigma layout of the unstructured configuration
LID = 0.05                      # lid velocity of the cavities
CHANNELS = 24                   # the surrogate's width


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest run: a grid of test size, ten steps; launches and
        # synchronisations count, not bandwidth
        {"name": "jacobi_f64_tiny", "kind": "jacobi", "cell": "f64", "nx": 24, "ny": 20, "nz": 16, "steps": 10},
        # heat diffusion as configured: 128^3 IEEE doubles, 100 steps
        {"name": "jacobi_f64_128", "kind": "jacobi", "cell": "f64", "nx": 128, "ny": 128, "nz": 128, "steps": 100},
        # the headline grid: 512^3 doubles held in fixed point, 100 steps
        {"name": "jacobi_fix_512", "kind": "jacobi", "cell": "fix", "nx": 512, "ny": 512, "nz": 512, "steps": 100},
        # an ordinary FP32 grid whose extents fit no tile
        {"name": "jacobi_f32_ragged", "kind": "jacobi", "cell": "f32", "nx": 325, "ny": 243, "nz": 187, "steps": 100},
        # Game of Life as configured: 8192^2 torus, 1000 generations
        {"name": "gol_8192", "kind": "gol", "nx": 8192, "ny": 8192, "torus": True, "steps": 1000},
        # a board of no particular size (rows not a multiple of a word)
        {"name": "gol_ragged", "kind": "gol", "nx": 1001, "ny": 777, "torus": True, "steps": 300},
        # unstructured diffusion as configured: 4.19 M nodes, 200 steps, FP64
        {"name": "sell_4m_f64", "kind": "sell", "n": 4194304, "precision": 8, "exact": False, "steps": 200},
        # a matrix that fits the caches, FP32, node count off the chunk size
        {"name": "sell_100k_f32", "kind": "sell", "n": 100003, "precision": 4, "exact": False, "steps": 200},
        # an uneven ensemble of lid-driven cavities, tuned, 1000 steps
        {"name": "lbm_8_f32", "kind": "lbm", "count": 8, "emin": 32, "emax": 128, "precision": 4, "tuned": True,
         "steps": 1000},
        # the surrogate's plain stencil: one judged segment on the 256^3 torus
        {"name": "varcoef_f32_256", "kind": "varcoef", "nx": 256, "ny": 256, "nz": 256, "precision": 4, "steps": 128},
        # the network advancing the 256^3 field (32 plain steps' worth)
        {"name": "surrogate_256", "kind": "advance", "nx": 256, "ny": 256, "nz": 256, "calls": 2},
        # one rank's share of a training iteration: 64^3 tori, batch 8
        {"name": "train_64_b8", "kind": "train", "nx": 64, "ny": 64, "nz": 64, "batch": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jacobi", "jacobi", "gol", "sell", "lbm", "varcoef", "advance", "train"])
    if kind == "jacobi":
        cell = rng.choice(["f64", "fix", "f32"])
        hi = 160 if cell == "f64" else 448
        return {"kind": kind, "cell": cell, "nx": _log_int(rng, 16, hi), "ny": _log_int(rng, 12, hi),
                "nz": _log_int(rng, 10, hi), "steps": _log_int(rng, 10, 100)}
    if kind == "gol":
        nx = _log_int(rng, 48, 8192)
        if rng.random() < 0.4:
            nx = max(64, nx // 32 * 32)
        return {"kind": kind, "nx": nx, "ny": _log_int(rng, 48, 8192), "torus": rng.random() < 0.8,
                "steps": _log_int(rng, 50, 300)}
    if kind == "sell":
        return {"kind": kind, "n": _log_int(rng, 2000, 3000000), "precision": rng.choice([8, 8, 4]),
                "exact": rng.random() < 0.3, "steps": _log_int(rng, 20, 200)}
    if kind == "lbm":
        emin = rng.randint(16, 48)
        return {"kind": kind, "count": rng.randint(1, 10), "emin": emin, "emax": rng.randint(emin, 112),
                "precision": rng.choice([4, 4, 8]), "tuned": rng.random() < 0.5, "steps": _log_int(rng, 50, 500)}
    if kind == "varcoef":
        precision = rng.choice([4, 4, 8])
        hi = 256 if precision == 4 else 128
        nx = _log_int(rng, 24, hi)
        if rng.random() < 0.5:
            nx = max(32, nx // 32 * 32)
        return {"kind": kind, "nx": nx, "ny": _log_int(rng, 24, hi), "nz": _log_int(rng, 24, hi),
                "precision": precision, "steps": 16 * rng.randint(1, 8)}
    if kind == "advance":
        return {"kind": kind, "nx": 32 * rng.randint(1, 8), "ny": 4 * rng.randint(8, 64), "nz": rng.randint(24, 256),
                "calls": rng.randint(1, 2)}
    return {"kind": kind, "nx": 32 * rng.randint(1, 2), "ny": 4 * rng.randint(8, 16), "nz": rng.randint(24, 64),
            "batch": rng.randint(1, 8)}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _uniform(shape, seed, salt, dtype=torch.float64):
    return torch.rand(shape, generator=_gen(seed, salt), device="cuda", dtype=dtype)


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _smooth(shape, seed, salt, lo, hi, length=16.0):
    """Periodic Gaussian random fields on tori (..., nz, ny, nx), each mapped
    to [lo, hi], FP32: the surrogate's fields and coefficients."""
    noise = torch.randn(shape, generator=_gen(seed, salt), device="cuda")
    nz, ny, nx = shape[-3:]
    kz, ky = (2 * math.pi * torch.fft.fftfreq(n, device="cuda") for n in (nz, ny))
    kx = 2 * math.pi * torch.fft.rfftfreq(nx, device="cuda")
    k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2
    f = torch.fft.irfftn(torch.fft.rfftn(noise, dim=(-3, -2, -1)) * torch.exp(-0.5 * k2 * length * length),
                         s=(nz, ny, nx), dim=(-3, -2, -1))
    a, b = f.amin(dim=(-3, -2, -1), keepdim=True), f.amax(dim=(-3, -2, -1), keepdim=True)
    return (lo + (hi - lo) * (f - a) / (b - a)).contiguous()


def _grid_values(case, seed):
    """Initial cells of a structured run, (nz, ny, nx) or (ny, nx)."""
    if case["kind"] == "gol":
        return (_uniform((case["ny"], case["nx"]), seed, 1, torch.float32) < 0.3).to(torch.uint8)
    dt = torch.float32 if case["cell"] == "f32" else torch.float64
    return _uniform((case["nz"], case["ny"], case["nx"]), seed, 1, dt)


def _graph(n, seed):
    """Random directed graph in CSR: out-degrees from a power law truncated
    to [4, 64], uniform targets, weights of a row summing to 0.9."""
    u = _uniform((n,), seed, 2)
    deg = torch.clamp(torch.floor(4.0 / (1.0 - u * (1.0 - 4.0 / 65.0))), 4, 64).to(torch.int64)
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row_ptr[1:] = torch.cumsum(deg, 0)
    nnz = int(row_ptr[-1])
    col = torch.randint(0, n, (nnz,), generator=_gen(seed, 3), device="cuda", dtype=torch.int32)
    w = _uniform((nnz,), seed, 4)
    w = 0.9 * w / torch.repeat_interleave(torch.segment_reduce(w, "sum", lengths=deg), deg)
    return row_ptr, col, w


def _cavities(case, seed):
    """Edges spread over the case's range (the program's), relaxation rates
    drawn per run."""
    edges = np.random.default_rng(42).integers(case["emin"], case["emax"] + 1, case["count"]).astype(np.int32)
    return edges, np.random.default_rng(int(seed) + 77).uniform(1.0, 1.9, case["count"])


def _params(seed):
    """Network parameters with a trained network's small increments (about
    a hundredth of the field): He initialisation, last layer scaled down."""
    p = surrogate.init_params(CHANNELS, int(seed) % 1000003)
    p[-(27 * CHANNELS + 1):] *= 0.1
    return p


def _fields(case, seed):
    shape = ((case["batch"],) if "batch" in case else ()) + (case["nz"], case["ny"], case["nx"])
    return _smooth(shape, seed, 5, 0.0, 1.0), _smooth(shape, seed, 6, 0.02, 0.15)


def _diffuse(u, k, steps):
    """Plain steps of the variable-coefficient stencil on tori by torch."""
    for _ in range(steps):
        flux = torch.zeros_like(u)
        for axis in (-1, -2, -3):
            for shift in (1, -1):
                flux += 0.5 * (k + torch.roll(k, shift, axis)) * (torch.roll(u, shift, axis) - u)
        u = u + flux
    return u


def _increment(u, k):
    """What a surrogate call is trained to give: 16 plain steps' change."""
    return (_diffuse(u, k, surrogate.STEPS_PER_CALL) - u).contiguous()


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("jacobi", "gol"):
        if kind == "gol":
            cell, periodic = lgd.CELL_GOL_U8, 3 if case["torus"] else 0
        else:
            cell, periodic = {"f64": lgd.CELL_JACOBI7_F64, "fix": lgd.CELL_JACOBI7_F64_FIX,
                              "f32": lgd.CELL_JACOBI7_F32}[case["cell"]], 0
        s["in"] = _pinned(_grid_values(case, seed))
        s["out"] = torch.empty(s["in"].shape, dtype=s["in"].dtype, pin_memory=True)
        s["grid"] = lgd.Grid(cell, tuple(s["in"].shape), periodic=periodic)
    elif kind == "sell":
        row_ptr, col, w = _graph(case["n"], seed)
        torch.cuda.synchronize()            # the library reads the arrays on a stream of its own
        s["grid"] = lgd.SellGrid.from_csr(case["n"], row_ptr, col, w, CHUNK, SIGMA, precision=case["precision"],
                                          exact=case["exact"], device=True)
        s["in"] = _pinned(_uniform((case["n"],), seed, 7))
        s["out"] = torch.empty(case["n"], dtype=torch.float64, pin_memory=True)
        if case["precision"] == 4:
            s["out32"] = torch.empty(case["n"], dtype=torch.float32)
    elif kind == "lbm":
        edges, omegas = _cavities(case, seed)
        s["ens"] = lgd.LbmEnsemble(edges, omegas, lid=LID, precision=case["precision"])
        if case["tuned"]:
            s["ens"].tune(4)
        shapes = [(19, int(e), int(e), int(e)) for e in edges]
        s["out"] = [torch.empty(sh, dtype=torch.float64, pin_memory=True) for sh in shapes]
        if case["precision"] == 4:
            s["out32"] = [torch.empty(sh, dtype=torch.float32) for sh in shapes]
    elif kind == "varcoef":
        dt = torch.float32 if case["precision"] == 4 else torch.float64
        u, k = (t.to(dt).contiguous() for t in _fields(case, seed))
        s["plain"] = surrogate.PlainStencil(precision=case["precision"], shape=(case["nz"], case["ny"], case["nx"]))
        s["plain"].set_kappa(k)
        s["in"], s["u"] = u, torch.empty_like(u)
    elif kind == "advance":
        s["in"], s["kappa"] = _fields(case, seed)
        s["u"] = torch.empty_like(s["in"])
        s["net"] = surrogate.SurrogateNet((case["nz"], case["ny"], case["nx"]), channels=CHANNELS)
        s["net"].set_params(_params(seed))
        s["stream"] = torch.cuda.ExternalStream(s["net"].stream())
        torch.cuda.synchronize()            # the fields are ready for the network's stream
    else:
        s["in"], s["kappa"] = _fields(case, seed)
        s["target"] = _increment(s["in"], s["kappa"])
        s["du"] = torch.empty_like(s["in"])
        s["net"] = surrogate.SurrogateNet((case["nz"], case["ny"], case["nx"]), batch=case["batch"],
                                          channels=CHANNELS, training=True)
        s["net"].set_params(_params(seed))
        s["stream"] = torch.cuda.ExternalStream(s["net"].stream())
        torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("jacobi", "gol"):
        s["grid"].upload(0, s["in"].numpy())
        s["grid"].step(case["steps"])
        s["grid"].download(0, out=s["out"].numpy())
        return s["out"]
    if kind == "sell":
        s["grid"].upload(s["in"].numpy())
        s["grid"].step(case["steps"])
        s["grid"].download(out=s["out"].numpy())
        if case["precision"] == 4:          # kept in the precision it was computed in
            return s["out32"].copy_(s["out"])
        return s["out"]
    if kind == "lbm":
        ens = s["ens"]
        ens.reset()
        ens.step(case["steps"])
        for j, out in enumerate(s["out"]):
            lgd.check(lgd.lib().lgd_lbm_download(ens._h, j, ctypes.c_void_p(out.data_ptr()), out.numel() * 8))
        if case["precision"] == 4:
            return [a.copy_(b) for a, b in zip(s["out32"], s["out"])]
        return s["out"]
    if kind == "varcoef":
        s["u"].copy_(s["in"])
        s["plain"].run(s["u"], case["steps"])
        return s["u"]
    net = s["net"]
    if kind == "advance":
        with torch.cuda.stream(s["stream"]):
            s["u"].copy_(s["in"])
        net.advance(s["u"], s["kappa"], case["calls"])
        return s["u"]
    # forward, loss and gradients; the ranks of a data-parallel run exchange
    # gradient and loss in BF16, the network's own precision
    net.forward(s["in"], s["kappa"], s["du"])
    loss = net.backward(s["target"])
    grads = torch.from_numpy(net.get_grads()).to(torch.bfloat16)
    with torch.cuda.stream(s["stream"]):
        s["du"] += s["in"]                  # the predicted fields
    return {"u": s["du"], "grads": grads, "loss": torch.tensor(loss, dtype=torch.bfloat16)}


# -------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "sell":
        # expected entries of the degree distribution (mean of the truncated law)
        nnz = case["n"] * 11.4
        p = case["precision"]
        return {"bytes": nnz * (p + 4) + case["n"] * 16.0, "flops": 2.0 * nnz * case["steps"]}
    if kind == "lbm":
        edges, _ = _cavities(dict(case), 1)
        cells = float(sum(int(e) ** 3 for e in edges))
        return {"bytes": cells * 19 * 2 * case["precision"], "flops": cells * case["steps"] * 250.0}
    cells = float(case["nx"]) * case["ny"] * case.get("nz", 1) * case.get("batch", 1)
    if kind == "gol":
        return {"bytes": 2.0 * cells, "flops": 0.0}
    if kind == "jacobi":
        return {"bytes": cells * (8 if case["cell"] == "f32" else 16), "flops": 7.0 * cells * case["steps"]}
    if kind == "varcoef":
        return {"bytes": 3.0 * cells * case["precision"], "flops": 31.0 * cells * case["steps"]}
    if kind == "advance":
        return {"bytes": 12.0 * cells, "flops": float(surrogate.FLOP_PER_VOXEL) * cells * case["calls"]}
    # forward, input gradients of layers 2 .. 4, weight gradients of all
    f = float(surrogate.FLOP_PER_VOXEL)
    return {"bytes": 16.0 * cells, "flops": cells * (3.0 * f - 2 * 27 * 2 * CHANNELS)}


# ------------------------------------------------------------------- exact
def _conv(h, w, b):
    """Periodic 3^3 convolution of channels-last fields [..., z, y, x, c] in
    their own precision; w [27][cin][cout], taps z slowest."""
    out = b.expand(h.shape[:-1] + (w.shape[2],))
    for tap in range(27):
        d = (tap // 9 - 1, tap // 3 % 3 - 1, tap % 3 - 1)
        out = out + torch.roll(h, tuple(-v for v in d), dims=(-4, -3, -2)) @ w[tap]
    return out


def _split_params(flat):
    out, off = [], 0
    for ci, co in ((2, CHANNELS), (CHANNELS, CHANNELS), (CHANNELS, CHANNELS), (CHANNELS, 1)):
        out.append((flat[off:off + 27 * ci * co].view(27, ci, co), flat[off + 27 * ci * co:off + 27 * ci * co + co]))
        off += 27 * ci * co + co
    return out


def _net(u, k, flat):
    h = torch.stack([u, k], dim=-1)
    layers = _split_params(flat)
    for i, (w, b) in enumerate(layers):
        h = _conv(h, w, b)
        if i < 3:
            h = torch.nn.functional.gelu(h)
    return h[..., 0]


_E = [(0, 0, 0), (0, 1, 0), (1, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (-1, -1, 0),
      (1, 1, 0), (1, -1, 0), (-1, 0, 1), (-1, 0, -1), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1), (0, -1, 1),
      (0, -1, -1)]                           # D3Q19 directions (x, y, z)
_OPP = [_E.index(tuple(-v for v in e)) for e in _E]


def _cavity(L, omega, steps):
    """D3Q19 BGK lid-driven cavity, pull scheme with half-way bounce-back."""
    dev = dict(device="cuda", dtype=torch.float64)
    w = torch.tensor([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, **dev).view(19, 1)
    e = torch.tensor(_E, **dev)
    coords = torch.arange(L, device="cuda")
    cell = torch.arange(L ** 3, device="cuda").view(L, L, L)
    src, add = [], torch.zeros((19, L ** 3), **dev)
    for i, (ex, ey, ez) in enumerate(_E):
        z, y, x = torch.meshgrid(coords - ez, coords - ey, coords - ex, indexing="ij")
        inside = (x >= 0) & (x < L) & (y >= 0) & (y < L) & (z >= 0) & (z < L)
        idx = torch.where(inside, i * L ** 3 + (z * L + y) * L + x, _OPP[i] * L ** 3 + cell)
        src.append(idx.reshape(-1))
        if ey == -1 and ex != 0:
            lid = (~inside) & (coords.view(1, L, 1) == L - 1)
            add[i] = torch.where(lid, 6.0 / 36.0 * ex * LID, 0.0).reshape(-1)
    src = torch.stack(src)
    f = w.expand(19, L ** 3).contiguous()
    eq = torch.where(torch.arange(19, device="cuda") == 0, 1 / 3, torch.where(
        torch.arange(19, device="cuda") < 7, 1 / 18, 1 / 36)).to(torch.float64).view(19, 1)
    for _ in range(steps):
        f = f.reshape(-1)[src] + add
        rho = f.sum(0)
        u = e.t() @ f
        eu = e @ u
        base = rho - 1.5 * (u * u).sum(0)
        f = (1.0 - omega) * f + omega * eq * (base + 3.0 * eu + 4.5 * eu * eu)
    return f.view(19, L, L, L)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gol":
        return None                         # whole numbers
    if kind == "jacobi":
        u = _grid_values(case, seed).double()
        for _ in range(case["steps"]):
            p = torch.nn.functional.pad(u, (1, 1, 1, 1, 1, 1))
            u = u + p[1:-1, :-2, 1:-1]
            u += p[1:-1, 2:, 1:-1]
            u += p[1:-1, 1:-1, 2:]
            u += p[1:-1, 1:-1, :-2]
            u += p[2:, 1:-1, 1:-1]
            u += p[:-2, 1:-1, 1:-1]
            u *= 1.0 / 7.0
        return u
    if kind == "sell":
        row_ptr, col, w = _graph(case["n"], seed)
        m = torch.sparse_csr_tensor(row_ptr, col.to(torch.int64), w, (case["n"], case["n"]))
        x = _uniform((case["n"],), seed, 7)
        for _ in range(case["steps"]):
            x = 0.1 * x + m @ x
        return x
    if kind == "lbm":
        edges, omegas = _cavities(case, seed)
        if sum(int(L) ** 3 for L in edges) * case["steps"] > 1e10:
            return None
        return [_cavity(int(L), float(o), case["steps"]) for L, o in zip(edges, omegas)]
    u, k = _fields(case, seed)
    if kind == "varcoef":
        return _diffuse(u.double(), k.double(), case["steps"])
    flat = torch.from_numpy(_params(seed)).cuda().double()
    if kind == "advance":
        u, k = u.double(), k.double()
        for _ in range(case["calls"]):
            u = u + _net(u, k, flat)
        return u
    flat.requires_grad_(True)
    u64, k64 = u.double(), k.double()
    du = _net(u64, k64, flat)
    loss = ((du - _increment(u, k).double()) ** 2).mean()
    loss.backward()
    return {"u": (u64 + du).detach(), "grads": flat.grad, "loss": loss.detach()}
