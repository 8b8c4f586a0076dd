"""The measured work of this library: solves as a user's program issues them.

Every case goes through the package's public entry points on 6-DOF lattice
systems (one 6x6 stiffness block per edge of a side^3 node lattice, the model
of the repository's own generator): plain solves over the range of sides the
tests and the benchmark use (4 to 80), refined solves, batches, a served burst,
the reference's driver on general CSR systems, its arithmetic, and single SpMV
calls. Inputs are made here from the seed alone.
"""
import math

import numpy as np
import torch

import wgpu_solver_backend_b200 as wsb


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest solve a program makes: 64 nodes, inputs on the device.
        # Launches and reduction latency are all of its time.
        dict(name="solve_tiny", kind="solve", side=4, host=False, tol=1e-6, aniso=0.0),
        # A small model from host arrays, as a script calls Matrix.solve.
        dict(name="solve_small_host", kind="solve", side=9, host=True, tol=1e-6, aniso=0.0),
        # An everyday model (29,478 unknowns) inside a device program.
        dict(name="solve_medium", kind="solve", side=17, host=False, tol=1e-6, aniso=0.0),
        # A larger model (196,608 unknowns), stiffness contrast of 10.
        dict(name="solve_ordinary", kind="solve", side=32, host=False, tol=1e-6, aniso=0.5),
        # The benchmark's largest system: 80^3 nodes, 3,072,000 unknowns.
        dict(name="solve_largest", kind="solve", side=80, host=False, tol=1e-6, aniso=0.0),
        # One request of the served workload alone: strong anisotropy, FP64
        # refinement to a true relative residual of 1e-8.
        dict(name="refined", kind="refined", side=21, tol=1e-8, aniso=2.0),
        # The opt-in single-reduction recurrence.
        dict(name="single_reduction", kind="single_reduction", side=40, tol=1e-6, aniso=0.0),
        # The reference's driver with its executors on a general CSR system:
        # supports take away unknowns, so blocks have 1 to 6 rows and n is odd
        # as often as not.
        dict(name="driver_csr", kind="driver", side=19, tol=1e-6, aniso=0.0, supports=0.03),
        # The same driver in the reference's own FP32 arithmetic (parity runs).
        dict(name="driver_reference_f32", kind="reference", side=12, tol=1e-6, aniso=0.0, supports=0.03),
        # Many independent systems of mixed sizes solved together.
        dict(name="batch", kind="batch", count=48, side_min=4, side_max=24, tol=1e-6, aniso=0.0),
        # A burst of requests to the server, host arrays in and out, each
        # refined to 1e-8 (the benchmark's end-to-end workload, smaller sides).
        dict(name="server_burst", kind="server", count=24, side_min=4, side_max=32, tol=1e-8, aniso=2.0),
        # One y = A x of a resident matrix, as a residual check issues it.
        dict(name="spmv", kind="spmv", side=41, layout="bsr6"),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "refined", "single_reduction", "driver", "reference", "batch",
                       "server", "spmv"])
    if kind == "solve":
        return dict(kind=kind, side=_log_int(rng, 4, 72), host=rng.random() < 0.4, tol=rng.choice([1e-5, 1e-6]),
                    aniso=round(rng.uniform(0.0, 1.0), 2))
    if kind == "refined":
        return dict(kind=kind, side=_log_int(rng, 4, 40), tol=rng.choice([1e-6, 1e-8, 1e-10]),
                    aniso=round(rng.uniform(0.0, 2.0), 2))
    if kind == "single_reduction":
        return dict(kind=kind, side=_log_int(rng, 4, 56), tol=1e-6, aniso=round(rng.uniform(0.0, 1.0), 2))
    if kind == "driver":
        return dict(kind=kind, side=_log_int(rng, 4, 36), tol=1e-6, aniso=round(rng.uniform(0.0, 1.0), 2),
                    supports=round(math.exp(rng.uniform(math.log(0.01), math.log(0.4))), 3))
    if kind == "reference":
        return dict(kind=kind, side=_log_int(rng, 4, 22), tol=1e-6, aniso=0.0,
                    supports=round(math.exp(rng.uniform(math.log(0.01), math.log(0.4))), 3))
    if kind == "batch":
        lo = rng.randint(3, 8)
        return dict(kind=kind, count=_log_int(rng, 4, 64), side_min=lo, side_max=rng.randint(lo + 4, 24), tol=1e-6,
                    aniso=round(rng.uniform(0.0, 1.0), 2))
    if kind == "server":
        lo = rng.randint(4, 8)
        return dict(kind=kind, count=_log_int(rng, 4, 24), side_min=lo, side_max=rng.randint(lo + 4, 30), tol=1e-8,
                    aniso=round(rng.uniform(0.5, 2.0), 2))
    return dict(kind="spmv", side=_log_int(rng, 4, 72), layout=rng.choice(["bsr6", "csr"]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _lattice(side, seed, aniso, supports=0.0):
    """Row pointers, columns, values (FP32 CSR, sorted columns), block starts
    and right-hand side of a side^3 lattice, as tensors on the device. Every
    edge carries S = R R^T / 6 + 0.1 I with R ~ N(0, 1), scaled by
    10^U(-aniso, aniso); 1e-3 I is added on the diagonal. `supports`: the share
    of nodes that lose 1 to 5 of their 6 unknowns."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1000003 + side)
    nodes = side ** 3
    V = torch.zeros(side, side, side, 6, 7, 6, device=dev)  # z, y, x, row, neighbour, column
    M = torch.zeros(side, side, side, 7, dtype=torch.bool, device=dev)
    M[..., 3] = True
    V[..., 3, :] += 1e-3 * torch.eye(6, device=dev)
    # Neighbours in column order: -z, -y, -x, self, +x, +y, +z.
    for axis, (lo, hi) in enumerate(((0, 6), (1, 5), (2, 4))):
        shape = [side, side, side]
        shape[axis] = side - 1
        R = torch.randn(*shape, 6, 6, generator=gen, device=dev)
        S = torch.matmul(R, R.transpose(-1, -2)) / 6.0
        S = 0.5 * (S + S.transpose(-1, -2)) + 0.1 * torch.eye(6, device=dev)
        u = torch.rand(*shape, 1, 1, generator=gen, device=dev)
        S = S * torch.pow(10.0, aniso * (2.0 * u - 1.0))
        first = [slice(None)] * 3
        second = [slice(None)] * 3
        first[axis] = slice(0, side - 1)
        second[axis] = slice(1, side)
        first, second = tuple(first), tuple(second)
        for at, nb in ((first, hi), (second, lo)):
            V[at + (slice(None), 3, slice(None))] += S
            V[at + (slice(None), nb, slice(None))] = -S
            M[at + (nb,)] = True
    V = V.view(nodes, 6, 7, 6)
    M = M.view(nodes, 7)
    keep = torch.ones(nodes, 6, dtype=torch.bool, device=dev)
    if supports > 0.0:
        # As many nodes for every seed, losing 1, 2, 3, 4, 5, 1, ... unknowns.
        cut = torch.rand(nodes, generator=gen, device=dev).argsort()[: int(round(supports * nodes))]
        lost = torch.zeros(nodes, dtype=torch.long, device=dev)
        lost[cut] = 1 + torch.arange(cut.numel(), device=dev) % 5
        order = torch.rand(nodes, 6, generator=gen, device=dev).argsort(dim=1).argsort(dim=1)
        keep = order >= lost[:, None]
    number = (torch.cumsum(keep.view(-1).long(), 0) - 1).view(nodes, 6)
    off = torch.tensor([-side * side, -side, -1, 0, 1, side, side * side], device=dev)
    nb = (torch.arange(nodes, device=dev)[:, None] + off).clamp(0, nodes - 1)
    entry = (M[:, None, :, None] & keep[:, :, None, None] & keep[nb][:, None, :, :]).expand(nodes, 6, 7, 6)
    val = V[entry]
    col = number[nb][:, None, :, :].expand(nodes, 6, 7, 6)[entry].to(torch.int32)
    per_row = entry.view(nodes, 6, 42).sum(dim=2)[keep]
    row_ptr = torch.zeros(per_row.numel() + 1, dtype=torch.int32, device=dev)
    row_ptr[1:] = torch.cumsum(per_row, 0)
    starts = torch.zeros(nodes + 1, dtype=torch.int32, device=dev)
    starts[1:] = torch.cumsum(keep.sum(dim=1), 0)
    n = per_row.numel()
    b = 2.0 * torch.rand(n, generator=gen, device=dev) - 1.0
    return dict(n=n, row_ptr=row_ptr, col=col, val=val, starts=starts, b=b)


def _sides(case):
    """The sides of a batch or burst: spread over the logarithm of the range,
    in mixed order."""
    u = np.random.default_rng(case["count"]).permutation((np.arange(case["count"]) + 0.5) / case["count"])
    lo, hi = math.log(case["side_min"]), math.log(case["side_max"] + 1)
    return [min(case["side_max"], int(math.exp(lo + x * (hi - lo)))) for x in u]


def _host(t, pinned=False):
    a = t.cpu()
    if pinned and torch.cuda.is_available():
        a = a.pin_memory()
    a = a.numpy()
    return a.view(np.uint32) if a.dtype == np.int32 else a


def _systems(case, seed):
    if case["kind"] in ("batch", "server"):
        return [_lattice(s, seed + 17 * i, case["aniso"]) for i, s in enumerate(_sides(case))]
    return [_lattice(case["side"], seed, case.get("aniso", 0.0), case.get("supports", 0.0))]


_MAX_ITER = 60000


def prepare(case, seed):
    kind = case["kind"]
    ctx = wsb.GpuContext.create("auto")
    systems = _systems(case, seed)
    st = dict(kind=kind, ctx=ctx, case=case)
    if kind == "server":
        # Requests in pinned host memory; the server borrows them and prepares
        # each on the GPU (the configuration the benchmark serves with).
        st["requests"] = [tuple(_host(s[k], True) for k in ("row_ptr", "col", "val", "starts", "b")) for s in systems]
        st["server"] = wsb.Server(ctx, borrow_inputs=True, device_prep=True)
        return st
    arrays = [tuple(_host(s[k]) for k in ("row_ptr", "col", "val", "starts", "b")) for s in systems]
    if kind in ("driver", "reference"):
        rp, ci, v, bs, b = arrays[0]
        n = len(rp) - 1
        lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
        st.update(n=n, b=b, spmv=wsb.SpmvExecutor.create(ctx, n, rp, ci, v), vec=wsb.VecOpsExecutor.create(ctx),
                  dot=wsb.DotScalarExecutor.create(ctx, n, 7), bj=wsb.BlockJacobiExecutor.create(ctx, n, lu, bs),
                  up=wsb.PcgUpdateScalarsExecutor.create(ctx))
        return st
    layout = wsb.LAYOUT_CSR if case.get("layout") == "csr" else wsb.LAYOUT_AUTO
    st["matrices"] = [wsb.Matrix.create(ctx, rp, ci, v, bs, layout=layout) for rp, ci, v, bs, _ in arrays]
    st["rhs"] = [a[4] for a in arrays]
    if kind in ("solve", "refined", "single_reduction", "spmv") and not case.get("host"):
        # Device vectors on a stream that the program shares with the library.
        st["stream"] = torch.cuda.Stream()
        ctx.set_stream(st["stream"].cuda_stream)
        st["b"] = systems[0]["b"]
        st["x"] = torch.zeros_like(st["b"])
        torch.cuda.synchronize()
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind in ("solve", "refined", "single_reduction"):
        m = state["matrices"][0]
        kw = dict(max_iter=_MAX_ITER, rel_tol=case["tol"])
        if kind == "refined":
            kw = dict(max_iter=_MAX_ITER, rel_tol=0.0, precision=wsb.PREC_MIXED_F64_IR, target_relres=case["tol"],
                      inner_rel_tol=1e-4)
        if kind == "single_reduction":
            kw["algorithm"] = wsb.ALG_SINGLE_REDUCTION
        if case.get("host"):
            return m.solve(state["rhs"][0], **kw)[0]
        with torch.cuda.stream(state["stream"]):
            state["x"].zero_()
            m.solve_device(state["b"].data_ptr(), state["x"].data_ptr(), **kw)
        return state["x"]
    if kind in ("driver", "reference"):
        x = np.zeros(state["n"], np.float32)
        wsb.pcg_block_jacobi_csr_wgpu(state["n"], state["b"], x, _MAX_ITER, case["tol"], 0.0, state["ctx"],
                                      state["spmv"], state["vec"], state["dot"], state["bj"], state["up"],
                                      precision=wsb.PREC_REFERENCE_F32 if kind == "reference"
                                      else wsb.PREC_F32_F64DOT)
        return x
    if kind == "batch":
        bt = wsb.Batch(state["ctx"])
        ids = [bt.add(m, b, max_iter=_MAX_ITER, rel_tol=case["tol"]) for m, b in zip(state["matrices"], state["rhs"])]
        bt.solve()
        return [bt.result(i, m.n)[0] for i, m in zip(ids, state["matrices"])]
    if kind == "server":
        srv = state["server"]
        rids = [srv.submit(*r, max_iter=_MAX_ITER, rel_tol=0.0, precision=wsb.PREC_MIXED_F64_IR,
                           target_relres=case["tol"], inner_rel_tol=1e-4) for r in state["requests"]]
        return [srv.wait(r)[0] for r in rids]
    with torch.cuda.stream(state["stream"]):
        state["matrices"][0].spmv_device(state["b"].data_ptr(), state["x"].data_ptr())
    return state["x"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _iterations(side, tol, aniso):
    """About how many iterations such a solve takes (lattice diameter and
    contrast set the condition number, up to the 1e-3 shift)."""
    its = min(40.0 * side ** 0.75, 470.0) * (1.0 + aniso) * math.log10(1.0 / tol) / 6.0
    return max(8.0, its)


def work(case):
    if case["kind"] in ("batch", "server"):
        sides = _sides(case)
    else:
        sides = [case["side"]]
    total_b = total_f = 0.0
    for s in sides:
        n = 6 * s ** 3
        blocks = s ** 3 + 6 * s * s * (s - 1)
        general = case.get("supports", 0.0) > 0.0 or case.get("layout") == "csr"
        keep = 1.0 - 0.5 * case.get("supports", 0.0)
        n *= keep
        matrix = blocks * 36 * keep * keep * (8.0 if general else 148.0 / 36.0)
        nnz = blocks * 36 * keep * keep
        if case["kind"] == "spmv":
            total_b += matrix + 8.0 * n
            total_f += 2.0 * nnz
            continue
        # Matrix, factors (24 bytes a row), right-hand side and solution once.
        total_b += matrix + 24.0 * n + 8.0 * n
        # Per iteration: product, block solve, three updates, three dots.
        total_f += _iterations(s, case["tol"], case["aniso"]) * (2.0 * nnz + 24.0 * n)
    return {"bytes": total_b, "flops": total_f}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _csr64(s):
    return torch.sparse_csr_tensor(s["row_ptr"].long(), s["col"].long(), s["val"].double(), size=(s["n"], s["n"]))


def _solution64(s, deadline_iters=20000):
    """A^-1 b in 64 bits: dense below 4,000 unknowns, else CG with the block
    diagonal, to a relative residual of 1e-13."""
    A, b, n = _csr64(s), s["b"].double(), s["n"]
    if n <= 4000:
        return torch.linalg.solve(A.to_dense(), b)
    # Inverse diagonal blocks, padded to 6x6 with the identity.
    starts = s["starts"].long()
    size = starts[1:] - starts[:-1]
    nodes = size.numel()
    node_of = torch.repeat_interleave(torch.arange(nodes, device=b.device), size)
    row = torch.repeat_interleave(torch.arange(n, device=b.device), (s["row_ptr"][1:] - s["row_ptr"][:-1]).long())
    col = s["col"].long()
    same = node_of[row] == node_of[col]
    D = torch.eye(6, dtype=torch.float64, device=b.device).repeat(nodes, 1, 1)
    at = node_of[row[same]]
    D[at, row[same] - starts[at], col[same] - starts[at]] = s["val"][same].double()
    D = torch.linalg.inv(D)
    place = torch.arange(n, device=b.device) - starts[node_of]
    del row, col, same, at

    def precondition(r):
        p = torch.zeros(nodes, 6, 1, dtype=torch.float64, device=b.device)
        p[node_of, place, 0] = r
        return torch.matmul(D, p)[node_of, place, 0]

    x = torch.zeros_like(b)
    for _ in range(3):  # restarts on the true residual
        r = b - A @ x
        z = precondition(r)
        p, rz = z.clone(), torch.dot(r, z)
        stop = 1e-13 * float(torch.linalg.norm(b))
        for k in range(deadline_iters):
            if k % 50 == 0 and float(torch.linalg.norm(r)) <= stop:
                break
            q = A @ p
            alpha = rz / torch.dot(p, q)
            x = x + alpha * p
            r = r - alpha * q
            z = precondition(r)
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
    return x


def exact(case, seed):
    systems = _systems(case, seed)
    if case["kind"] == "spmv":
        return _csr64(systems[0]) @ systems[0]["b"].double()
    if case["kind"] == "reference":
        # FP32 arithmetic throughout: its distance to the solution is its own.
        return _solution64(systems[0])
    out = [_solution64(s) for s in systems]
    return out if case["kind"] in ("batch", "server") else out[0]
