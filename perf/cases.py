"""The inversions that are timed: what a user of this framework has it do.

A case is one call (or one short sequence of calls) of the public entry points
on block p-cyclic matrices of p x p blocks of n x n:

  invert   device-resident inversion of an assembled matrix (a DQMC walker
           that keeps its matrices on the GPU)
  dqmc     matrix from expm(K) and the auxiliary fields, inversion, and
           sign / log|det| for the acceptance ratio, all on the device
  split    factorization + R^{-1} and the explicit inverse as two calls, with
           the state between them read (the determinant's sign is in it)
  mixed    inversion with the products on the int8 tensor cores
  batch    independent walkers of several lattice sizes in one call
  handle   the handle API on page-locked host arrays, float64 or float32

Matrices are the Hubbard model's on lx x ly periodic lattices (n = lx ly), or
general ones with dense random blocks.  Every pass starts from the packed
blocks, since the inversions overwrite their matrix.
"""
import math

import numpy as np
import torch

from bsofi_b200 import api, fp32
from bsofi_b200.flops import bsofi_flops
from bsofi_b200.hubbard import expm_sym

DTAU = 0.125


def listed():
    return [
        # The smallest lattices of the tests: a call is launches and latency.
        {"name": "invert_4x4_p8", "kind": "invert", "lx": 4, "ly": 4, "p": 8, "U": 4.0},
        # A general matrix of odd sizes: ragged tiles, unaligned columns.
        {"name": "invert_random_n37_p19", "kind": "invert", "n": 37, "p": 19},
        # The smallest benchmark configuration.
        {"name": "invert_8x8_p16", "kind": "invert", "lx": 8, "ly": 8, "p": 16, "U": 4.0},
        # The single-precision library as a host program calls it.
        {"name": "handle32_8x8_p16", "kind": "handle", "single": True, "lx": 8, "ly": 8, "p": 16,
         "U": 4.0},
        # A host program's call, copies included.
        {"name": "handle_10x10_p32", "kind": "handle", "lx": 10, "ly": 10, "p": 32, "U": 4.0},
        # A mid-size lattice through the two-call form.
        {"name": "split_12x12_p20", "kind": "split", "lx": 12, "ly": 12, "p": 20, "U": 4.0},
        # A DQMC sweep step at low temperature (many time slices).
        {"name": "dqmc_10x10_p64", "kind": "dqmc", "lx": 10, "ly": 10, "p": 64, "U": 4.0},
        # Walkers of several lattice sizes together (sides 8..16, p 8..64).
        {"name": "batch_16_mixed_sizes", "kind": "batch", "count": 16, "U": 4.0, "mix": 3},
        # The headline configuration.
        {"name": "invert_16x16_p32", "kind": "invert", "lx": 16, "ly": 16, "p": 32, "U": 4.0},
        {"name": "mixed_16x16_p32", "kind": "mixed", "lx": 16, "ly": 16, "p": 32, "U": 4.0},
        # Blocks as large as the serving stream's largest, few time slices.
        {"name": "invert_24x24_p12", "kind": "invert", "lx": 24, "ly": 24, "p": 12, "U": 4.0},
        # The largest single inversion (5.2 GB matrix).
        {"name": "invert_20x20_p64", "kind": "invert", "lx": 20, "ly": 20, "p": 64, "U": 6.0},
    ]


def draw(rng):
    kind = rng.choice(["invert", "invert", "invert", "dqmc", "split", "mixed", "handle", "batch"])
    u = rng.choice([2.0, 4.0, 6.0])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 20), "U": u, "mix": rng.randrange(1 << 16)}
    most = {"mixed": 9000, "handle": 3200}.get(kind, 12000)
    while True:
        case = {"kind": kind}
        if kind in ("invert", "split") and rng.random() < 0.4:
            case["n"] = n = int(round(math.exp(rng.uniform(math.log(8), math.log(576)))))
        else:
            case["lx"] = rng.randint(3, 24)
            case["ly"] = rng.randint(max(3, case["lx"] - 4), min(24, case["lx"] + 4))
            case["U"] = u
            n = case["lx"] * case["ly"]
        case["p"] = p = int(round(math.exp(rng.uniform(math.log(3), math.log(96)))))
        if kind == "handle" and rng.random() < 0.4:
            case["single"] = True
        if n * p <= most:
            return case


# ------------------------------------------------------------------ inputs
def _size(case):
    return (case["n"] if "n" in case else case["lx"] * case["ly"]), case["p"]


def _instances(case):
    """The cases of a batch: sides 8..16, p 8..64, as its mix number says."""
    r = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        side = int(r.integers(8, 17))
        out.append({"lx": side, "ly": side, "p": int(r.integers(8, 65)), "U": case["U"]})
    return out


def _exp_hopping(lx, ly):
    """expm(dtau K) of the periodic lx x ly lattice's adjacency K (symmetric)."""
    def ring(m):
        a = np.zeros((m, m))
        for i in range(m):
            for j in (i - 1, (i + 1) % m):
                if j % m != i:
                    a[i, j % m] = 1.0
        return a
    k = np.kron(ring(lx), np.eye(ly)) + np.kron(np.eye(lx), ring(ly))
    return expm_sym(DTAU * k)


def _lam(case):
    return math.acosh(math.exp(case["U"] * DTAU / 2.0))


def _fields(case, seed):
    n, p = _size(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 2, (p, n), generator=g, device="cuda").double() * 2 - 1


def _blocks(case, seed):
    """(diagonal blocks or None for identities, coupling blocks), each block
    column-major: T[k, j, i] is element (i, j) of block k."""
    n, p = _size(case)
    if "n" in case:
        g = torch.Generator(device="cuda").manual_seed(seed)
        d = torch.randn(p, n, n, dtype=torch.float64, device="cuda", generator=g)
        d += torch.eye(n, dtype=torch.float64, device="cuda")
        return d, torch.randn(p, n, n, dtype=torch.float64, device="cuda", generator=g)
    e = torch.from_numpy(_exp_hopping(case["lx"], case["ly"])).cuda()
    b = e.T.unsqueeze(0) * torch.exp(_lam(case) * _fields(case, seed)).unsqueeze(2)
    b[: p - 1].neg_()
    return None, b.contiguous()


def _dense(d, s, dtype=torch.float64):
    """The matrix column-major on the GPU: T[j, i] is element (i, j)."""
    p, n, _ = s.shape
    t = torch.zeros(n * p, n * p, dtype=dtype, device="cuda")
    eye = torch.eye(n, dtype=dtype, device="cuda")
    for k in range(p):
        c = slice(k * n, (k + 1) * n)
        r = (k + 1) % p
        t[c, c] = eye if d is None else d[k]
        t[c, r * n:(r + 1) * n] = s[k]
    return t


def _device_state(case, seed, ws_bytes):
    n, p = _size(case)
    N = n * p
    return {"n": n, "p": p, "N": N, "A": torch.empty(N, N, dtype=torch.float64, device="cuda"),
            "tau": torch.empty(N, dtype=torch.float64, device="cuda"),
            "ws": torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for i, c in enumerate(_instances(case)):
            s = _device_state(c, 0, 0)
            s["d"], s["s"] = _blocks(c, seed * 1000 + i)
            parts.append(s)
        ns, ps, ld = [q["n"] for q in parts], [q["p"] for q in parts], [q["N"] for q in parts]
        ws = torch.empty(api.batch_workspace_bytes(ns, ps, ld), dtype=torch.uint8, device="cuda")
        return {"kind": kind, "parts": parts, "ns": ns, "ps": ps, "ld": ld, "ws": ws}
    n, p = _size(case)
    N = n * p
    if kind == "handle":
        np_type, t_type = (np.float32, torch.float32) if case.get("single") else (np.float64, torch.float64)
        d, s = _blocks(case, seed)
        keep = torch.empty(N, N, dtype=t_type, pin_memory=True)
        tau = torch.empty(N, dtype=t_type, pin_memory=True)
        h = (fp32 if case.get("single") else api).Handle(n, p)
        return {"kind": kind, "n": n, "p": p, "keep": (keep, tau), "A": keep.numpy().T,
                "tau": tau.numpy(), "h": h, "work": np.zeros(max(1, h.lwork()), dtype=np_type),
                "d": None if d is None else d.to(t_type).cpu().numpy(),
                "s": s.to(t_type).cpu().numpy(), "eye": np.eye(n, dtype=np_type)}
    mixed = kind == "mixed"
    st = _device_state(case, seed, api.mixed_workspace_bytes(n, p, N) if mixed
                       else api.workspace_bytes(n, p, N))
    st["kind"] = kind
    if kind == "dqmc":
        st["e"] = torch.from_numpy(_exp_hopping(case["lx"], case["ly"])).cuda()  # symmetric
        st["h"] = _fields(case, seed)
        st["lam"] = _lam(case)
        st["det"] = torch.empty(2, dtype=torch.float64, device="cuda")
    else:
        st["d"], st["s"] = _blocks(case, seed)
    return st


# ------------------------------------------------------------------ one pass
def _ok(rc):
    if rc != 0:
        raise RuntimeError("call failed (%d)" % rc)


def _assemble(s, stream):
    _ok(api.device_assemble(s["n"], s["p"], 0 if s["d"] is None else s["d"].data_ptr(),
                            s["s"].data_ptr(), s["A"].data_ptr(), s["N"], stream))


def run(state):
    kind = state["kind"]
    if kind == "handle":
        return _run_handle(state)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "batch":
        for s in state["parts"]:
            _assemble(s, stream)
        _ok(api.device_invert_batched(state["ns"], state["ps"],
                                      [s["A"].data_ptr() for s in state["parts"]], state["ld"],
                                      [s["tau"].data_ptr() for s in state["parts"]],
                                      state["ws"].data_ptr(), streams=16, stream=stream))
        return {"inverse": [s["A"] for s in state["parts"]],
                "tau": [s["tau"] for s in state["parts"]]}
    n, p, N, A, tau = state["n"], state["p"], state["N"], state["A"], state["tau"]
    a = (n, p, A.data_ptr(), N, tau.data_ptr(), state["ws"].data_ptr())
    if kind == "dqmc":
        _ok(api.device_hubbard_assemble(n, p, state["e"].data_ptr(), state["h"].data_ptr(),
                                        state["lam"], A.data_ptr(), N, stream))
        _ok(api.device_bsoftri(*a, stream))
        _ok(api.device_logdet(n, p, A.data_ptr(), N, tau.data_ptr(), 1, state["det"].data_ptr(),
                              stream))
        _ok(api.device_bsoi(*a, stream))
        return {"inverse": A, "tau": tau, "det": state["det"]}
    _assemble(state, stream)
    if kind == "split":
        _ok(api.device_bsoftri(*a, stream))
        # The state a caller reads between the two calls: R^{-1}'s diagonal
        # and last block column (the determinant and equal-time quantities).
        diag, last = torch.diagonal(A).clone(), A[(p - 1) * n:].clone()
        _ok(api.device_bsoi(*a, stream))
        return {"inverse": A, "tau": tau, "diag": diag, "last": last}
    if kind == "mixed":
        _ok(api.device_invert_mixed(*a, 0, stream))
    else:
        _ok(api.device_invert(*a, stream))
    return {"inverse": A, "tau": tau}


def _run_handle(state):
    """The caller writes the blocks into its array, then the two calls."""
    n, p, A = state["n"], state["p"], state["A"]
    t = A.T
    for k in range(p):
        c = slice(k * n, (k + 1) * n)
        r = (k + 1) % p
        t[c, c] = state["eye"] if state["d"] is None else state["d"][k]
        t[c, r * n:(r + 1) * n] = state["s"][k]
    h = state["h"]
    _ok(h.bsoftri(A, state["tau"], state["work"]))
    _ok(h.bsoi(A, state["tau"], state["work"]))
    return {"inverse": t, "tau": state["tau"]}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: the nonzero blocks read, the inverse and tau written.  Flops: the
    LAPACK operation counts of the factorization, R^{-1} and the products."""
    if case["kind"] == "batch":
        each = [work(dict(c, kind="invert")) for c in _instances(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n, p = _size(case)
    N = n * p
    inputs = N + n * n if case["kind"] == "dqmc" else (2 if "n" in case else 1) * p * n * n
    return {"bytes": (4.0 if case.get("single") else 8.0) * (inputs + N * N + N),
            "flops": float(bsofi_flops(n, p))}


# ------------------------------------------------------------------ values
def _exact_one(d, s):
    """Inverse and tau of the structured QR: (inverse column-major, tau, R^{-1}
    diagonal and last block column) from torch's LU and Householder QR."""
    p, n, _ = s.shape
    t = _dense(d, s)
    inv = torch.linalg.inv(t.T.contiguous()).T.contiguous()
    N = n * p
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    blk = lambda k: (eye if d is None else d[k].T)  # noqa: E731
    tau = torch.empty(N, dtype=torch.float64, device="cuda")
    R = torch.zeros(N, N, dtype=torch.float64, device="cuda")
    head, corner = blk(0), s[p - 1].T  # A(k, k) and A(k, p-1) before panel k
    for k in range(p - 2):
        q, tk = torch.geqrf(torch.cat([head, s[k].T]))
        rest = torch.zeros(2 * n, 2 * n, dtype=torch.float64, device="cuda")
        rest[n:, :n] = blk(k + 1)
        rest[:n, n:] = corner
        rest = torch.ormqr(q, tk, rest, left=True, transpose=True)
        tau[k * n:(k + 1) * n] = tk
        R[k * n:(k + 1) * n, k * n:(k + 1) * n] = torch.triu(q[:n])
        R[k * n:(k + 1) * n, (k + 1) * n:(k + 2) * n] = rest[:n, :n]
        R[k * n:(k + 1) * n, (p - 1) * n:] = rest[:n, n:]
        head, corner = rest[n:, :n], rest[n:, n:]
    k = p - 2
    q, tk = torch.geqrf(torch.cat([torch.cat([head, corner], 1),
                                   torch.cat([s[k].T, blk(p - 1)], 1)]))
    tau[k * n:] = tk
    R[k * n:, k * n:] = torch.triu(q)
    rhs = torch.zeros(N, n, dtype=torch.float64, device="cuda")
    rhs[(p - 1) * n:] = eye
    last = torch.linalg.solve_triangular(R, rhs, upper=True)
    last[(p - 1) * n:] += torch.tril(q, -1)[n:, n:]  # the reflectors stay below the diagonal
    return inv, tau, 1.0 / torch.diagonal(R), last.T.contiguous()


def exact(case, seed):
    if case["kind"] == "batch":
        each = [_exact_one(*_blocks(c, seed * 1000 + i)) for i, c in enumerate(_instances(case))]
        return {"inverse": [e[0] for e in each], "tau": [e[1] for e in each]}
    d, s = _blocks(case, seed)
    if case.get("single"):
        d, s = None if d is None else d.float().double(), s.float().double()
    inv, tau, diag, last = _exact_one(d, s)
    if case["kind"] == "split":
        return {"inverse": inv, "tau": tau, "diag": diag, "last": last}
    if case["kind"] == "dqmc":
        sign, log = torch.linalg.slogdet(_dense(d, s))
        return {"inverse": inv, "tau": tau, "det": torch.stack([sign, log])}
    return {"inverse": inv, "tau": tau}
