"""Performance cases of the framework: what a user has it do, through its public entry points.

The work is the pseudo-likelihood and its gradient (one evaluation, alone or
inside an optimizer), the sequence weights before it and the contact map after
it.  Sizes span what protein alignments have: tens to a thousand columns L,
hundreds to tens of thousands of rows N.

A case is a dict of plain values:

  kind "eval"      Evaluator.evaluate(x, g) on CUDA tensors: f to the host, g whole
  kind "host"      the same on (pinned) host arrays, x in and g out over PCIe
  kind "autograd"  f and its gradients through torch autograd
  kind "solve"     Evaluator.minimize: a number of conjugate-gradient iterations
  kind "batch"     solve_batch: a ragged batch from alignments to contact maps
  kind "weights"   calculate_weights: sequence weights from a host alignment

with the sizes "L" and "N" (for a batch: of its largest alignment) and, by kind,
"path", "iterations" and "count".
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ccmpred_b200 as ccm
from ccmpred_b200 import autograd, host

Q, QPAD = 21, 32


def listed():
    return [
        # the smallest families: a call is latency and launches
        dict(name="eval L50 N200", kind="eval", L=50, N=200, path="tc_i8sp"),
        # few rows on the path that the per-size table takes for them
        dict(name="eval L90 N600 bf16x2", kind="eval", L=90, N=600, path="tc_bf16x2"),
        # a domain of ordinary size
        dict(name="eval L150 N2000", kind="eval", L=150, N=2000, path="tc_i8sp"),
        # odd sizes: no multiple of a tile, a vector or a warp
        dict(name="eval L253 N7001", kind="eval", L=253, N=7001, path="tc_i8sp"),
        # the benchmark's alignment
        dict(name="eval L300 N5000", kind="eval", L=300, N=5000, path="tc_i8sp"),
        # the widest and deepest alignment of the benchmark
        dict(name="eval L1000 N20000", kind="eval", L=1000, N=20000, path="tc_i8sp"),
        # host-pointer callers (the shape of the reference's CPU evaluation)
        dict(name="host L180 N3000", kind="host", L=180, N=3000, path="tc_i8sp"),
        # differentiable use: true partial derivatives, forward and backward
        dict(name="autograd L150 N2000", kind="autograd", L=150, N=2000, path="tc_i8sp"),
        # a device-side solve of one family, from the bias start
        dict(name="solve L120 N1500", kind="solve", L=120, N=1500, iterations=12, path="tc_i8sp"),
        # many families at once, as a database is processed
        dict(name="batch 12 L<=200 N<=4000", kind="batch", L=200, N=4000, count=12, iterations=8,
             path="tc_i8sp"),
        # sequence weights before every run: an ordinary and a deep alignment
        dict(name="weights L300 N5000", kind="weights", L=300, N=5000),
        dict(name="weights L1000 N20000", kind="weights", L=1000, N=20000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval"] * 6 + ["host", "autograd", "solve", "batch", "weights", "weights"])
    if kind == "eval":
        path = rng.choice(["tc_i8sp"] * 5 + ["tc_bf16x2"])
        top = (400, 2000) if path == "tc_bf16x2" else (1000, 20000)
        return dict(kind=kind, L=_log_int(rng, 40, top[0]), N=_log_int(rng, 200, top[1]), path=path)
    if kind == "host":
        return dict(kind=kind, L=_log_int(rng, 60, 300), N=_log_int(rng, 300, 6000), path="tc_i8sp")
    if kind == "autograd":
        return dict(kind=kind, L=_log_int(rng, 40, 200), N=_log_int(rng, 200, 5000), path="tc_i8sp")
    if kind == "solve":
        return dict(kind=kind, L=_log_int(rng, 50, 400), N=_log_int(rng, 200, 10000),
                    iterations=rng.randint(8, 16), path="tc_i8sp")
    if kind == "batch":
        return dict(kind=kind, L=_log_int(rng, 80, 300), N=_log_int(rng, 800, 6000),
                    count=rng.randint(6, 16), iterations=rng.randint(6, 10), path="tc_i8sp")
    return dict(kind=kind, L=_log_int(rng, 50, 1000), N=_log_int(rng, 200, 20000))


# ------------------------------------------------------------------ inputs
def _msa(L, N, seed):
    """N x L states 0..20: column frequencies Dirichlet(0.5), 12 % gaps, and 30 %
    of the rows near-duplicates of others (5-25 % of their positions redrawn)."""
    rng = np.random.Generator(np.random.PCG64([seed, L, N]))
    cdf = np.cumsum(rng.dirichlet(np.full(Q - 1, 0.5), size=L), axis=1)
    grid = (np.arange(4096) + 0.5) / 4096
    table = np.stack([np.searchsorted(c, grid) for c in cdf]).clip(0, Q - 2).astype(np.uint8)
    table = table.reshape(-1)

    def cells(rows):
        u = rng.integers(0, 4096, size=(rows, L), dtype=np.int32)
        m = table[u + 4096 * np.arange(L, dtype=np.int32)]
        m[rng.random((rows, L), dtype=np.float32) < 0.12] = Q - 1
        return m

    msa = cells(N)
    dup = int(0.3 * N)
    if dup:
        src = rng.integers(0, N - dup, size=dup)
        redrawn = (rng.random((dup, L), dtype=np.float32) <
                   rng.uniform(0.05, 0.25, size=(dup, 1)).astype(np.float32))
        msa[N - dup:] = np.where(redrawn, msa[N - dup:], msa[src])
        msa = msa[rng.permutation(N)]
    return np.ascontiguousarray(msa)


def _fields(L, seed):
    """V ~ N(0, 0.1), W ~ N(0, 0.01) with W(b,k,a,j) = W(a,j,b,k) and zero self
    blocks, on the GPU: V as (20, L), W as (21, L, 21, L) in the order b, k, a, j."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + L)
    V = torch.randn(Q - 1, L, generator=gen, device="cuda") * 0.1
    W = torch.randn(Q * L, Q * L, generator=gen, device="cuda").mul_(0.01).triu_(1)
    W += W.T.clone()
    W = W.view(Q, L, Q, L)
    i = torch.arange(L, device="cuda")
    W[:, i, :, i] = 0.0
    return V, W


def _padded(V, W):
    L = V.shape[1]
    x = torch.zeros(ccm.nvar_padded(L), device=V.device, dtype=V.dtype)
    x[: (Q - 1) * L] = V.reshape(-1)
    x[ccm.nsingle_padded(L):].view(Q, L, QPAD, L)[:, :, :Q] = W
    return x


def _batch_sizes(case):
    """Sizes of a batch: spread over L/4 .. L and N/20 .. N, the largest among them."""
    out = []
    for i in range(case["count"]):
        u, v = (i * 0.618034) % 1.0, (i * 0.754878) % 1.0
        out.append((int(round(case["L"] * (1 - 0.75 * u))), int(round(case["N"] * 20.0 ** -v))))
    return out


# ------------------------------------------------------------------ cases
def prepare(case, seed):
    kind, L, N = case["kind"], case["L"], case["N"]
    if kind == "batch":
        msas = [_msa(l, n, seed + 17 * i) for i, (l, n) in enumerate(_batch_sizes(case))]
        return dict(case=case, msas=msas)
    msa = _msa(L, N, seed)
    if kind == "weights":
        return dict(case=case, msa=msa)
    w = ccm.calculate_weights(msa, 0.8)
    ev = ccm.Evaluator(msa, weights=w, path=case["path"],
                       gradient="partial" if kind == "autograd" else "tied")
    state = dict(case=case, ev=ev)
    if kind == "solve":
        state["x0"] = torch.from_numpy(host.init_bias(msa)).cuda()
        return state
    V, W = _fields(L, seed)
    if kind == "autograd":
        state["V"] = V.T.contiguous().requires_grad_()
        state["W"] = W.permute(1, 3, 0, 2).contiguous().requires_grad_()
        return state
    x = _padded(V, W)
    del V, W
    if kind == "host":
        pinned = torch.empty(x.numel(), pin_memory=True)
        pinned.copy_(x)
        state["x"] = pinned.numpy()
        state["g"] = torch.empty(x.numel(), pin_memory=True).numpy()
        return state
    state["x"] = x
    state["g"] = torch.empty_like(x)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("eval", "host"):
        f = state["ev"].evaluate(state["x"], state["g"])
        return f, state["g"]
    if kind == "autograd":
        V, W = state["V"], state["W"]
        f = autograd.pseudo_likelihood(V, W, state["ev"])
        gV, gW = torch.autograd.grad(f, (V, W))
        return f, gV, gW
    if kind == "solve":
        x = state["x0"].clone()
        r = state["ev"].minimize(x, max_iterations=case["iterations"], epsilon=1e-6)
        return r.fx, x
    if kind == "batch":
        res, maps = ccm.solve_batch(state["msas"], path=case["path"], epsilon=1e-6,
                                    max_iterations=case["iterations"])
        return [r.fx for r in res], maps
    return ccm.calculate_weights(state["msa"], 0.8)


# ------------------------------------------------------------------ what a pass cannot do without
def _eval_work(L, N):
    """One evaluation: the two contractions over the 21 L coupling columns; x and
    the alignment read, g written."""
    return 4.0 * N * (Q * L) ** 2, 8.0 * ccm.nvar_padded(L) + N * L + 4.0 * N


def work(case):
    kind, L, N = case["kind"], case["L"], case["N"]
    if kind == "weights":  # a comparison for every pair of rows and column
        return dict(flops=0.5 * N * N * L, bytes=N * L + 4.0 * N)
    flops, size = _eval_work(L, N)
    if kind == "solve":  # at least one evaluation at x0 and one for each iteration
        n = case["iterations"] + 1
        return dict(flops=n * flops, bytes=8.0 * ccm.nvar_padded(L) + N * L + 4.0 * N)
    if kind == "batch":
        flops = size = 0.0
        for l, n in _batch_sizes(case):
            flops += 0.5 * n * n * l + (case["iterations"] + 1) * _eval_work(l, n)[0]
            size += n * l + 4.0 * l * l
        return dict(flops=flops, bytes=size)
    if kind == "autograd":
        size = 8.0 * (L * (Q - 1) + (L * Q) ** 2) + N * L + 4.0 * N
    return dict(flops=flops, bytes=size)


# ------------------------------------------------------------------ 64-bit values
def _weights64(msa, threshold):
    """1 / (number of rows, the row itself counted twice, that agree with it in more
    than ceil(threshold L) columns - 1); the threshold product is taken in float."""
    N, L = msa.shape
    need = math.ceil(float(np.float32(threshold) * np.float32(L)))
    m = torch.from_numpy(msa).cuda()
    count = torch.ones(N, dtype=torch.float64, device="cuda")
    onehot = torch.zeros(N, Q * L, dtype=torch.float16, device="cuda")
    onehot.scatter_(1, (m.long() * L + torch.arange(L, device="cuda")), 1.0)
    for r in range(0, N, 2048):  # sums of at most L ones: whole numbers, exact in float32
        same = torch.matmul(onehot[r:r + 2048].float(), onehot.float().T) if N * Q * L < 5e8 else \
            sum(torch.matmul(onehot[r:r + 2048, c:c + 2100].float(), onehot[:, c:c + 2100].float().T)
                for c in range(0, Q * L, 2100))
        count[r:r + 2048] += (same > need).sum(1)
    return (1.0 / (count - 1.0)).cpu().numpy()


def _evaluate64(msa, weights, V, W, partial):
    """f, dV (20, L) and dW (21 L, 21 L; rows (b, k), columns (a, j)) in float64."""
    N, L = msa.shape
    QL = Q * L
    lam1, lam2 = float(np.float32(0.01)), float(np.float32(0.2) * np.float32(L - 1))
    V, M = V.double(), W.reshape(QL, QL).double()
    m = torch.from_numpy(msa).cuda().long()
    w = torch.from_numpy(np.asarray(weights, dtype=np.float64)).cuda()
    j = torch.arange(L, device="cuda")
    f = torch.zeros((), dtype=torch.float64, device="cuda")
    G1 = torch.zeros(QL, dtype=torch.float64, device="cuda")
    G2 = torch.zeros(QL, QL, dtype=torch.float64, device="cuda")
    bias = torch.cat([V, V.new_zeros(1, L)]).reshape(-1)
    for r in range(0, N, 4096):
        rows = m[r:r + 4096]
        O = torch.zeros(rows.shape[0], QL, dtype=torch.float64, device="cuda")
        O.scatter_(1, rows * L + j, 1.0)
        z = (O @ M + bias).view(-1, Q, L)
        lse = torch.logsumexp(z, 1)
        wr = w[r:r + 4096, None]
        f += (wr * (lse - z.gather(1, rows[:, None])[:, 0])).sum()
        R = (wr[:, None] * (torch.exp(z - lse[:, None]) - O.view(-1, Q, L))).reshape(-1, QL)
        G1 += R.sum(0)
        G2 += O.T @ R
        del O, z, R
    f += lam1 * (V * V).sum() + 0.5 * lam2 * (M * M).sum()
    dV = G1.view(Q, L)[: Q - 1] + 2.0 * lam1 * V
    if partial:
        return float(f), dV, G2 + lam2 * M
    G2 += G2.T.clone()
    G2.view(Q, L, Q, L)[:, j, :, j] = 0.0
    return float(f), dV, G2.add_(M, alpha=2.0 * lam2)


def exact(case, seed):
    kind, L, N = case["kind"], case["L"], case["N"]
    if kind in ("solve", "batch"):
        return None  # the end of an iteration: no closed value
    msa = _msa(L, N, seed)
    w = _weights64(msa, 0.8)
    if kind == "weights":
        return w
    V, W = _fields(L, seed)
    f, dV, dW = _evaluate64(msa, w.astype(np.float32), V, W, kind == "autograd")
    del V, W
    if kind == "autograd":
        return f, dV.T.contiguous(), dW.view(Q, L, Q, L).permute(1, 3, 0, 2).contiguous()
    return f, _padded(dV, dW.view(Q, L, Q, L))
