"""The measured workloads: what a prover built on this package has it do, through its public entry points.

`listed()` gives the fixed cases, `draw(rng)` more of the same ranges, `prepare(case, seed)` a case's inputs on the
GPU, `run(state)` one pass, `work(case)` the bytes and field operations a pass cannot do without, `tolerance(case)`
how far another correct implementation may be off (nothing: field elements and digests are whole numbers).

A case is a dict with a "kind":

  commit     Reed-Solomon encode of a batch of message rows, BLAKE3 column leaves, Merkle tree, in one shot (the
             coefficients too with "polys", as the prover keeps them for its later folds)
  committer  the same through RowCommitter, whose buffers a program keeps between commits
  stream     one commitment over rows that arrive in chunks, opened at queried columns, with their paths
  kquant     quantised weights lifted and encoded without the lifted matrix
  ntt        batched transforms in place, either direction
  sumcheck   product sumcheck, all challenges drawn beforehand
  gate       gate-shaped sumcheck (eq*a*b - eq*c), one challenge per round from a callback
  projection the proof of one matrix product: project both factors with challenges, then a sumcheck
  matmul     the witness product itself
  fold       rows of coefficients multiplied pairwise and summed in the evaluation domain
"""
import math

import numpy as np
import torch

from verinf_b200 import cuda_primitives as cp
from verinf_b200 import fold
from verinf_b200 import kquant_cuda as kq
from verinf_b200 import layergkr_gpu as lg
from verinf_b200.commit import RowCommitter, StreamCommitter

P = cp.P
DEV = "cuda"

# The production geometry: message slots, polynomial size, codeword length (the slots past ELL are the random pad).
ELL, K_DEG, N_LIG = 8192, 16384, 65536


def listed():
    return [
        # the smallest commitment in use: 64 rows of 2^10, no pad; launches and the tree's chain count
        dict(name="commit 64x2^10", kind="commit", rows=64, ell=1024, k=1024, n=4096, pad=False, polys=False),
        # one activation tensor (1000 x 4096 values) at the production geometry, coefficients kept
        dict(name="commit activation", kind="commit", rows=500, ell=ELL, k=K_DEG, n=N_LIG, pad=True, polys=True),
        # the large batch of the benchmark: 4096 x 2^16 -> 2^18 columns
        dict(name="commit 4096x2^16", kind="committer", rows=4096, ell=65536, k=65536, n=262144, pad=False),
        # one 5120 x 8192 expert weight in 1024-row chunks, 40 opened columns
        dict(name="stream expert", kind="stream", rows=5120, chunk=1024, ell=ELL, k=K_DEG, n=N_LIG, opened=40),
        # one MLP weight as Q4_K super-blocks, transposed as the loader has it
        dict(name="kquant Q4_K 11008x4096", kind="kquant", qtype="Q4_K", d_out=11008, d_in=4096, transpose=True),
        # a batch of message-sized transforms
        dict(name="ntt 64x2^16", kind="ntt", m=64, logn=16, inverse=False),
        # one long transform back to coefficients
        dict(name="intt 2^20", kind="ntt", m=1, logn=20, inverse=True),
        # three tables of 2^24, degree 3
        dict(name="sumcheck 3x2^24", kind="sumcheck", tables=3, logn=24),
        # a layer's gate batch, interactive
        dict(name="gate 2^18", kind="gate", logn=18),
        # the proof of an up-projection: X (1000 x 4096), W (4096 x 11008)
        dict(name="projection 4096x11008", kind="projection", seq=1000, n_in=4096, n_out=11008),
        # the witness of the same projection
        dict(name="matmul 1000x4096x11008", kind="matmul", m=1000, k=4096, n=11008),
        # a chunk of 1024 row pairs of the q_lin / p_0 folds
        dict(name="fold 1024x2^14", kind="fold", rows=1024, k=K_DEG),
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_geometry(rng, lo, hi):
    k = 1 << rng.randint(lo, hi)
    n = k * rng.choice((2, 4, 4, 4, 8))
    ell = rng.choice((k, k // 2, rng.randint(k // 2, k)))
    return ell, k, n


def draw(rng):
    kind = rng.choice(("commit", "commit", "committer", "stream", "kquant", "ntt", "ntt", "sumcheck", "gate",
                       "projection", "matmul", "matmul", "fold"))
    if kind in ("commit", "committer"):
        ell, k, n = _draw_geometry(rng, 8, 16)
        rows = _spread(rng, 16, min(6000, (1 << 28) // n))
        case = dict(kind=kind, rows=rows, ell=ell, k=k, n=n, pad=ell < k and rng.random() < 0.7)
        if kind == "commit":
            case["polys"] = rng.random() < 0.5
        return case
    if kind == "stream":
        ell, k, n = _draw_geometry(rng, 10, 15)
        rows = _spread(rng, 200, min(6000, (1 << 28) // n))
        return dict(kind=kind, rows=rows, chunk=rng.choice((256, 1000, 1024)), ell=ell, k=k, n=n,
                    opened=rng.randint(4, 80))
    if kind == "kquant":
        return dict(kind=kind, qtype=rng.choice(("Q4_K", "Q5_K", "Q6_K")), d_out=_spread(rng, 100, 11008),
                    d_in=256 * _spread(rng, 2, 16), transpose=rng.random() < 0.7)
    if kind == "ntt":
        logn = rng.randint(6, 22)
        return dict(kind=kind, m=_spread(rng, 1, max(1, min(3000, (1 << 24) >> logn))), logn=logn,
                    inverse=rng.random() < 0.5)
    if kind == "sumcheck":
        return dict(kind=kind, tables=rng.randint(2, 3), logn=rng.randint(8, 23))
    if kind == "gate":
        return dict(kind=kind, logn=rng.randint(8, 20))
    if kind == "projection":
        return dict(kind=kind, seq=_spread(rng, 1, 2000), n_in=_spread(rng, 64, 11008), n_out=_spread(rng, 64, 8192))
    if kind == "matmul":
        return dict(kind=kind, m=_spread(rng, 2, 1500), k=_spread(rng, 64, 11008), n=_spread(rng, 64, 4096))
    return dict(kind=kind, rows=_spread(rng, 5, 1024), k=1 << rng.randint(8, 14))


# ---- inputs ----------------------------------------------------------------------------------------------------
def _uniform(gen, *shape):
    """Uniform field elements: the high half below 2^32 - 1 keeps every value below p."""
    hi = torch.randint(0, (1 << 32) - 1, shape, dtype=torch.int64, device=DEV, generator=gen)
    lo = torch.randint(0, 1 << 32, shape, dtype=torch.int64, device=DEV, generator=gen)
    return hi.bitwise_left_shift_(32).bitwise_or_(lo).view(torch.uint64)


def _int8(gen, *shape):
    """int8 weights or activations in the field, negatives as p - |v|."""
    v = torch.randint(-128, 128, shape, dtype=torch.int64, device=DEV, generator=gen)
    return torch.where(v < 0, v + (P - (1 << 64)), v).view(torch.uint64)


def _seed32(gen):
    return torch.randint(0, 256, (32,), dtype=torch.uint8, device=DEV, generator=gen)


def _kquant_blocks(gen, qtype, d_out, d_in):
    """Super-blocks with random quants and sub-scales and fp16 scales of a trained weight's size."""
    raw = torch.randint(0, 256, (d_out * d_in // 256, kq.BLOCK_BYTES[qtype]), dtype=torch.uint8, device=DEV,
                        generator=gen)
    scale = (torch.randn((raw.size(0), 2), device=DEV, generator=gen) * 0.02).to(torch.float16).view(torch.uint8)
    if qtype == "Q6_K":
        raw[:, 208:210] = scale[:, :2]
    else:
        raw[:, 0:4] = scale
    return raw


def _coins(seed, n):
    rng = np.random.default_rng([7, seed])
    return [int(v) % P for v in rng.integers(0, 1 << 64, size=n, dtype=np.uint64)]


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("commit", "committer", "stream"):
        rows, ell = case["rows"], case["ell"]
        packed = ell < case["k"]            # with slots left for the pad the rows are packed int8 tensors
        s["msg"] = _int8(gen, rows, ell) if packed else _uniform(gen, rows, ell)
        s["seed"] = _seed32(gen) if case.get("pad", True) and packed else None
        if kind == "committer":
            s["plan"] = RowCommitter(rows, ell, case["k"], case["n"], master_seed=s["seed"])
        if kind == "stream":
            s["chunks"] = list(s["msg"].split(case["chunk"]))
            rng = np.random.default_rng([3, seed])
            s["cols"] = sorted(int(c) for c in rng.integers(0, case["n"], size=case["opened"]))
    elif kind == "kquant":
        s["raw"] = _kquant_blocks(gen, case["qtype"], case["d_out"], case["d_in"])
        s["seed"] = _seed32(gen)
    elif kind == "ntt":
        s["rows"] = _uniform(gen, case["m"], 1 << case["logn"])
    elif kind == "sumcheck":
        s["tables"] = [_uniform(gen, 1 << case["logn"]) for _ in range(case["tables"])]
        s["coins"] = _coins(seed, case["logn"])
    elif kind == "gate":
        s["tables"] = [_uniform(gen, 1 << case["logn"]) for _ in range(4)]
        s["coins"] = _coins(seed, case["logn"])
    elif kind == "projection":
        s["X"], s["W"] = _int8(gen, case["seq"], case["n_in"]), _int8(gen, case["n_in"], case["n_out"])
        s["rho"], s["tau"] = _uniform(gen, case["seq"]), _uniform(gen, case["n_out"])
        s["width"] = 1 << max(1, (case["n_in"] - 1).bit_length())
        s["coins"] = _coins(seed, s["width"].bit_length() - 1)
    elif kind == "matmul":
        s["X"], s["W"] = _int8(gen, case["m"], case["k"]), _int8(gen, case["k"], case["n"])
    elif kind == "fold":
        s["A"], s["B"] = _uniform(gen, case["rows"], case["k"]), _uniform(gen, case["rows"], case["k"])
        s["w"] = _uniform(gen, case["rows"])
    else:
        raise ValueError(kind)
    return s


# ---- passes ----------------------------------------------------------------------------------------------------
def _transcript(proof):
    """(claim, round polynomials, challenges, mask) as arrays of numbers."""
    claim, polys, _, _ = proof
    return np.array([claim], dtype=np.uint64), np.array([[y for _, y in r] for r in polys], dtype=np.uint64)


def _words(t):
    """Field elements as 64-bit words (int64 lanes), which torch can index."""
    return t.view(torch.int64)


def _run_commit(s):
    c = s["case"]
    if c["polys"]:
        polys, codes = cp.encode_rows(s["msg"], c["k"], c["n"], master_seed=s["seed"])
        root, levels = cp.merkle_build_blake3(cp.hash_columns_streamed(codes))
        return _words(polys), _words(codes), root, levels
    root, levels, codes = cp.commit_rows(s["msg"], c["k"], c["n"], master_seed=s["seed"])
    return _words(codes), root, levels


def _run_committer(s):
    p = s["plan"]
    root = p.commit(s["msg"])
    return root, _words(p.codes), p.leaves, p.upper


def _run_stream(s):
    c = s["case"]
    sc = StreamCommitter(c["rows"], c["ell"], c["k"], c["n"], master_seed=s["seed"], open_cols=s["cols"],
                         max_chunk_rows=c["chunk"])
    for chunk in s["chunks"]:
        sc.update(chunk)
    root = sc.finalize()
    return root, _words(sc.opened), sc.paths(), sc.upper


def _run_kquant(s):
    c = s["case"]
    return _words(kq.kquant_encode_rows(s["raw"], c["qtype"], 1 << 12, c["d_out"], c["d_in"], ell=ELL, k_deg=K_DEG,
                                        n_lig=N_LIG, transpose=c["transpose"], master_seed=s["seed"])[1])


def _run_ntt(s):
    (cp.ntt_inverse_batched if s["case"]["inverse"] else cp.ntt_forward_batched)(s["rows"])
    return _words(s["rows"])


def _run_sumcheck(s):
    coins = s["coins"]
    return _transcript(lg.prove_terms_gpu([(1, s["tables"])], lambda i: coins[i], coins=coins))


def _run_gate(s):
    eq, a, b, c = s["tables"]
    coins = s["coins"]
    return _transcript(lg.prove_terms_gpu([(1, [eq, a, b]), (P - 1, [eq, c])], lambda i: coins[i]))


def _run_projection(s):
    n_in, width, coins = s["case"]["n_in"], s["width"], s["coins"]
    a = cp.gl_matmul(s["rho"].reshape(1, -1), s["X"])[0]
    b = cp.gl_matvec(s["W"], s["tau"])
    tables = torch.zeros((2, width), dtype=torch.int64, device=DEV)
    tables[0, :n_in] = a.view(torch.int64)
    tables[1, :n_in] = b.view(torch.int64)
    tables = tables.view(torch.uint64)
    proof = lg.prove_terms_gpu([(1, [tables[0], tables[1]])], lambda i: coins[i], coins=coins)
    return (_words(a), _words(b)) + _transcript(proof)


def _run_matmul(s):
    return _words(cp.gl_matmul(s["X"], s["W"]))


def _run_fold(s):
    return _words(fold.fold_products_eval(s["A"], s["B"], s["w"]))


_RUN = {"commit": _run_commit, "committer": _run_committer, "stream": _run_stream, "kquant": _run_kquant,
        "ntt": _run_ntt, "sumcheck": _run_sumcheck, "gate": _run_gate, "projection": _run_projection,
        "matmul": _run_matmul, "fold": _run_fold}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------------------------
def _encode_ops(rows, k, n):
    """Field operations of one interpolation and n/k coset transforms of length k (3 per butterfly)."""
    return rows * (1 + n // k) * 1.5 * k * math.log2(k)


def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: field additions, subtractions and products (hashing
    is counted as the bytes that it reads)."""
    kind = case["kind"]
    if kind in ("commit", "committer"):
        rows, ell, k, n = case["rows"], case["ell"], case["k"], case["n"]
        out = n + (k if case.get("polys") else 0)
        return {"bytes": 8.0 * rows * (ell + out) + 64.0 * n, "flops": _encode_ops(rows, k, n)}
    if kind == "stream":
        rows, ell, k, n = case["rows"], case["ell"], case["k"], case["n"]
        return {"bytes": 8.0 * rows * (ell + case["opened"]) + 64.0 * n, "flops": _encode_ops(rows, k, n)}
    if kind == "kquant":
        rows = -(-case["d_out"] * case["d_in"] // ELL)
        raw = case["d_out"] * case["d_in"] // 256 * kq.BLOCK_BYTES[case["qtype"]]
        return {"bytes": raw + 8.0 * rows * N_LIG, "flops": _encode_ops(rows, K_DEG, N_LIG)}
    if kind == "ntt":
        n = 1 << case["logn"]
        return {"bytes": 16.0 * case["m"] * n, "flops": 1.5 * case["m"] * n * case["logn"]}
    if kind in ("sumcheck", "gate"):
        n = 1 << case["logn"]
        tables = case.get("tables", 4)
        # per pair of entries of the first round a fold (3) per table and the products at deg + 1 points; rounds halve
        return {"bytes": 8.0 * tables * n, "flops": n * (3.0 * tables + (tables + 1) * (2 * tables))}
    if kind == "projection":
        seq, n_in, n_out = case["seq"], case["n_in"], case["n_out"]
        return {"bytes": 8.0 * (seq * n_in + n_in * n_out + seq + n_out + 2 * n_in),
                "flops": 2.0 * (seq * n_in + n_in * n_out) + 18.0 * n_in}
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 8.0 * (m * k + k * n + m * n), "flops": 2.0 * m * k * n}
    if kind == "fold":
        rows, k, n = case["rows"], case["k"], 2 * case["k"]
        return {"bytes": 8.0 * (rows * (2 * k + 1) + n), "flops": rows * n * (2 * 1.5 * math.log2(n) + 3.0)}
    raise ValueError(kind)


def tolerance(case):
    return "exact"
