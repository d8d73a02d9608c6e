"""Benchmark of the commit hot path: RS-encoded Goldilocks elements per second.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl native|reference]

One step = one commit of the large-batch configuration (4096 rows x 2^16 uniform field
elements, blow-up 4 by coset NTT to 2^18 columns, BLAKE3 column leaves, Merkle root).
With N > 1 (launched by torchrun, one rank per GPU) every rank commits its own batch
of the same size -- independent commits, no data-path collective; the 32-byte roots are
all-gathered -- so the job is weak-scaled and `value` is the aggregate over all ranks.

The same JSON line carries, beside the headline:
  sharded_commit    ONE Merkle tree over the 4096 rows split over the N ranks (rows/N each;
                    sub-tree chaining values all-gathered over NCCL inside the timed region),
  sharded_sumcheck  the degree-3 sumcheck of three 2^24 tables sharded over the N ranks
                    (per-round partial sums all-reduced), challenges from the seeded transcript,
  e2e               the headline from pinned host rows, with the bare host-to-device copy time
                    of the same buffers beside it,
  and on rank 0 the second half of the metric: the 7B-layer commit + sumcheck seconds, the
  fused K-quant lift + encode, and (with --extra) the MoE expert commits.
At N = 1 the CPU leg (the oracle, all host threads) commits the same rows and recomputes the
sumcheck, K-quant and layer figures' checkable parts, so one run checks itself.

`--impl reference` times the CPU restatement of the reference algorithm (the oracle,
OpenMP over all host threads) on a bounded sample of the same workload.
"""
import argparse
import hashlib
import json
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

P = (1 << 64) - (1 << 32) + 1
METRIC = "RS-encoded Goldilocks elems/s"
UNIT = "elems/s"
SEED = 1234               # block b of the global message is drawn with seed SEED + b
SC_SEED = 0               # sumcheck tables use seeds SC_SEED, +1, +2; coins from Transcript(b"bench/sumcheck")
SC_LOG = 24


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="native", choices=["native", "reference"])
    ap.add_argument("--rows", type=int, default=4096)
    ap.add_argument("--log-k", type=int, default=16)
    ap.add_argument("--blowup", type=int, default=4)
    ap.add_argument("--cpu-rows", type=int, default=0, help="rows of the CPU sample (0 = auto)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline / self-check leg")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--h2d-slices", type=int, default=32,
                    help="slices of the end-to-end host-to-device copy (a slice is encoded and hashed when it lands)")
    ap.add_argument("--no-sharded", action="store_true", help="skip the sharded commit and sharded sumcheck blocks")
    ap.add_argument("--no-secondary", action="store_true",
                    help="skip the 7B-layer commit+sumcheck and the fused K-quant encode on rank 0")
    ap.add_argument("--extra", action="store_true",
                    help="also run the MoE expert commits, the field matmul and the fold workloads")
    ap.add_argument("--micro", choices=["matmul", "fold", "sumcheck", "int_pipes"],
                    help="run only one secondary kernel (1024 x 2048 x 2048 matmul, the fold of 1024 row pairs "
                         "at K = 16384, or the 2^24 x 3 degree-3 sumcheck) and print its figures; the cases the ncu "
                         "summaries use.  int_pipes builds bench_int_pipes.cu into build/int_pipes and runs it "
                         "(integer issue rates and field-primitive throughputs)")
    return ap.parse_args()


def peaks():
    f = ROOT / "MEASURED_PEAKS.json"
    if f.exists():
        d = json.loads(f.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def workload_name(a):
    return (f"large-batch commit: {a.rows} rows x 2^{a.log_k} uniform Goldilocks elems, blowup {a.blowup} "
            f"coset NTT to 2^{a.log_k + (a.blowup.bit_length() - 1)} cols, BLAKE3 column hash + Merkle root")


# ----------------------------------------------------------------------------- synthetic input
def block_rows(total_rows):
    """The global message is made of 8 seeded blocks (so that 1, 2, 4 or 8 ranks hold whole blocks)."""
    return -(-total_rows // 8)


def gen_rows(torch, dev, r0, r1, k, total_rows, seed0=SEED):
    """Rows [r0, r1) of the global message, canonical uniform field elements, on `dev`.  Block b
    (rows b*B .. (b+1)*B) depends on seed0 + b only, whoever generates it."""
    from verinf_b200 import _lib
    B = block_rows(total_rows)
    parts = []
    for b in range(r0 // B, -(-r1 // B) if r1 > r0 else r0 // B):
        lo, hi = b * B, min((b + 1) * B, total_rows)
        g = torch.Generator(device=dev)
        g.manual_seed(seed0 + b)
        blk = torch.randint(-(1 << 63), (1 << 63) - 1, (hi - lo, k), dtype=torch.int64, device=dev, generator=g)
        parts.append(blk[max(r0, lo) - lo:min(r1, hi) - lo])
    if not parts:
        return torch.empty((0, k), dtype=torch.uint64, device=dev)
    msg = (parts[0] if len(parts) == 1 else torch.cat(parts)).contiguous().view(torch.uint64)
    zero = torch.zeros(1, dtype=torch.uint64, device=dev)
    if msg.numel():
        _lib.check(_lib.LIB.vi_gl_binary_bcast(1, msg.data_ptr(), zero.data_ptr(), 1, msg.data_ptr(), msg.numel(),
                                              _lib.stream_ptr()))          # canonicalise: x >= p -> x - p
    return msg


def sumcheck_tables(torch, dev):
    tabs = torch.empty((3, 1 << SC_LOG), dtype=torch.int64, device=dev)
    for i in range(3):
        g = torch.Generator(device=dev)
        g.manual_seed(SC_SEED + i)
        tabs[i] = torch.randint(0, 1 << 62, (1 << SC_LOG,), dtype=torch.int64, device=dev, generator=g)
    return tabs.view(torch.uint64)


def sumcheck_coins():
    from verinf_b200.transcript import seeded_coins
    return seeded_coins(b"bench/sumcheck", SC_SEED, "sc", SC_LOG)


# ----------------------------------------------------------------------------- CPU arm
def cpu_threads():
    import oracle
    return oracle.set_threads(os.cpu_count() or 1)     # a launcher's OMP_NUM_THREADS=1 must not starve the CPU arm


def cpu_commit(msg_np, n, steps=1, warmup=0):
    """Times oracle.commit_rows (encode + column hash + Merkle) on the given rows; returns
    (cpu_baseline dict, seconds per pass, root bytes)."""
    import oracle
    threads = cpu_threads()
    rows = msg_np.shape[0]
    root = None
    for _ in range(warmup):
        oracle.commit_rows(msg_np, n)
    t0 = time.perf_counter()
    for _ in range(steps):
        root = oracle.commit_rows(msg_np, n)
    dt = (time.perf_counter() - t0) / steps
    return {"value": rows * n / dt, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"{rows} rows of the workload (encode + column hash + Merkle), C oracle with OpenMP on "
                      f"{threads} threads, {dt:.2f} s per pass"}, dt, root


def cpu_rows_np(a, rows):
    """`rows` rows of the workload generated on the host with numpy (the reference arm has no GPU to draw
    them from: same distribution as the GPU arm's rows, not the same values)."""
    import numpy as np
    rng = np.random.default_rng(SEED)
    return rng.integers(0, P, size=(rows, 1 << a.log_k), dtype=np.uint64)


def auto_cpu_rows(a, budget_s=15.0):
    """Pick a sample that takes roughly `budget_s` on this host: probe 4 rows, then scale."""
    _, dt, _ = cpu_commit(cpu_rows_np(a, 4), (1 << a.log_k) * a.blowup)
    rows = int(max(8, min(a.rows, budget_s / max(dt / 4, 1e-6))))
    return rows - rows % 4


def run_reference(a):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    n = (1 << a.log_k) * a.blowup
    rows = a.cpu_rows or max(8, auto_cpu_rows(a) // max(a.steps + a.warmup, 1))
    base, dt, _ = cpu_commit(cpu_rows_np(a, rows), n, steps=a.steps, warmup=a.warmup)
    line = {
        "metric": METRIC, "value": base["value"], "unit": UNIT, "n_gpus": a.gpus, "steps": a.steps,
        "warmup": a.warmup, "ms_per_step": dt * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "u64", "data": "synthetic", "impl": "reference",
        "config": {"workload": workload_name(a), "sample_rows_per_step": rows},
        "cpu_baseline": dict(base),
        "e2e": {"value": base["value"], "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line))


def cpu_self_check(a, torch, msg_dev, root_hex, k, n, payload):
    """CPU leg at N = 1 (the only place of the native arm that touches the oracle): times the oracle on the
    SAME rows the GPU committed and requires the same root; recomputes the sumcheck transcript, sampled
    rows of the fused K-quant encode and the 7B-layer W_Q commitment + sumcheck from the payloads the GPU
    workloads returned."""
    import numpy as np
    import oracle
    out = {}
    crow = a.cpu_rows or auto_cpu_rows(a, budget_s=60.0)
    sample = msg_dev[:crow].view(torch.int64).cpu().numpy().view(np.uint64)
    base, _, root = cpu_commit(sample, n)
    if crow == a.rows:
        ok = root.hex() == root_hex
        base["sample"] += "; all rows of the GPU arm's batch, root equal: " + str(ok)
        out["commit_root_equals_oracle"] = ok
        assert ok, f"GPU root {root_hex} differs from the oracle's {root.hex()} on the same {crow} rows"
    else:
        from verinf_b200 import cuda_primitives as cp
        got, _, _ = cp.commit_rows(msg_dev[:crow].contiguous(), k, n)
        ok = bytes(got.cpu().tolist()) == root
        base["sample"] += f"; the first {crow} rows of the GPU arm's batch, prefix root equal: {ok}"
        out["commit_prefix_root_equals_oracle"] = ok
        assert ok, f"GPU root of the first {crow} rows differs from the oracle's"
    out["cpu_baseline"] = base
    sc = payload.get("sumcheck")
    if sc is not None:
        t0 = time.perf_counter()
        claim, samples, _ = oracle.sumcheck(sc["tables"], [(1, [0, 1, 2])], sc["coins"])
        dt = time.perf_counter() - t0
        ok = claim == sc["claim"] and [[int(v) for v in row[:4]] for row in samples] == sc["polys"]
        out["sumcheck_transcript_equals_oracle"] = ok
        out["sumcheck_cpu_s"] = dt
        assert ok, "2^24 x 3 sumcheck transcript differs from the oracle's"
    for kq in payload.get("kquant", []):
        w = oracle.kquant_to_field(kq["raw"], kq["qtype"], float(kq["S"]))
        rows = np.ascontiguousarray(w.reshape(kq["d_out"], kq["d_in"]).T).reshape(-1, kq["ell"])   # transposed, packed
        ok = True
        for i, r in enumerate(kq["rows"]):
            padded = np.empty((1, kq["k"]), dtype=np.uint64)
            padded[0, :kq["ell"]] = rows[r]
            padded[0, kq["ell"]:] = oracle.row_prg(kq["seed"], r, 1, kq["k"] - kq["ell"])
            ok = ok and np.array_equal(oracle.encode_rows(padded, kq["n"], want_polys=False)[1][0], kq["codes"][i])
        out.setdefault("kquant_rows_equal_oracle", {})[kq["qtype"]] = bool(ok)
        assert ok, f"fused {kq['qtype']} lift+encode differs from the oracle on rows {kq['rows']}"
    ly = payload.get("layer7b")
    if ly is not None:
        flat = ly["W_Q"].reshape(-1)
        m = flat.size // ly["ell"]
        padded = np.empty((m, ly["k"]), dtype=np.uint64)
        padded[:, :ly["ell"]] = flat.reshape(m, ly["ell"])
        padded[:, ly["ell"]:] = oracle.row_prg(ly["seed"], 0, m, ly["k"] - ly["ell"])
        ok_root = oracle.commit_rows(padded, ly["n"]) == ly["root_W_Q"]
        a_vec = oracle.gl_matmul(ly["rho"].reshape(1, -1), ly["X_Q"])[0]          # rho^T X
        b_vec = oracle.gl_matmul(ly["W_Q"], ly["tau"].reshape(-1, 1))[:, 0]       # W tau
        claim, samples, _ = oracle.sumcheck(np.stack([a_vec, b_vec]), [(1, [0, 1])], ly["coins"])
        ok_sc = claim == ly["claim"] and [[int(v) for v in row[:3]] for row in samples] == ly["polys"]
        out["layer7b_W_Q_root_equals_oracle"] = bool(ok_root)
        out["layer7b_W_Q_sumcheck_equals_oracle"] = bool(ok_sc)
        assert ok_root and ok_sc, "7B-layer W_Q commitment or sumcheck differs from the oracle"
    mo = payload.get("moe")
    if mo is not None:
        m = mo["msg"].shape[0]
        padded = np.empty((m, mo["k"]), dtype=np.uint64)
        padded[:, :mo["ell"]] = mo["msg"]
        padded[:, mo["ell"]:] = oracle.row_prg(mo["seed"], 0, m, mo["k"] - mo["ell"])
        ok = oracle.commit_rows(padded, mo["n"]) == mo["root"]
        out["moe_prefix_root_equals_oracle"] = bool(ok)
        assert ok, "MoE expert prefix commitment differs from the oracle"
    return out


# ----------------------------------------------------------------------------- GPU arm
class ClockSampler:
    """nvidia-smi clock and throttle-reason samples every 20 ms, started before the warm-up steps (the tool takes
    a few hundred ms to deliver its first line); stop(t0, t1) keeps the samples stamped inside the timed region,
    or, when the region was too short to hold two, those from the warm-up on (the GPU is under the same load)."""
    FIELDS = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.path = tempfile.NamedTemporaryFile(prefix="clocks_", suffix=".csv", delete=False).name
        self.proc = None
        self.idx = gpu_index

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.idx), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "20"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self, t0=None, t1=None):
        import datetime
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        if self.proc is None:
            return out
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in open(self.path).read().splitlines():
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 10:
                continue
            try:
                ts = datetime.datetime.strptime(f[0], "%Y/%m/%d %H:%M:%S.%f")
                rows.append((ts, float(f[2]), float(f[3]), [nm for nm, v in zip(names, f[6:10]) if v.lower().startswith("active")]))
            except ValueError:
                continue
        try:
            os.unlink(self.path)
        except OSError:
            pass
        window = "timed region"
        inside = [r for r in rows if t0 is not None and t0 <= r[0] <= t1]
        if len(inside) < 2:
            inside, window = [r for r in rows if t1 is None or r[0] <= t1], "warm-up and timed region"
        if inside:
            sm = sorted(r[1] for r in inside)
            out.update(sm_mhz=sm[len(sm) // 2], sm_max_mhz=max(r[2] for r in inside),
                       reasons=sorted({x for r in inside for x in r[3]}), samples=len(inside), window=window)
        return out


def all_agree(torch, dist, world, dev, ok: bool) -> bool:
    """Every rank learns whether a check held on all ranks (so nobody is left waiting in a collective)."""
    t = torch.tensor([1 if ok else 0], dtype=torch.int64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MIN)
    return bool(int(t.item()))


def run_native(a):
    import torch
    import torch.distributed as dist

    from verinf_b200 import _lib
    from verinf_b200 import distributed as D
    from verinf_b200.commit import RowCommitter

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; the native arm has no CPU fallback")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    numa_bound = D.bind_to_gpu_numa(local)          # pinned host rows next to the GPU that reads them
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)

    k, n, rows = 1 << a.log_k, (1 << a.log_k) * a.blowup, a.rows
    # rank r's own batch = blocks 8r .. 8r+7 of the seeded stream; rank 0's batch is also the global
    # message of the sharded commit
    msg = gen_rows(torch, dev, 0, rows, k, rows, seed0=SEED + 8 * rank)
    com = RowCommitter(rows, k, k, n, device=dev, h2d_slices=a.h2d_slices)
    roots = [torch.empty(32, dtype=torch.uint8, device=dev) for _ in range(world)] if world > 1 else None

    def step():
        root = com.commit(msg)
        if world > 1:
            dist.all_gather(roots, root.contiguous())
        return root

    def fence():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    import datetime
    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()
    for _ in range(max(a.warmup, 3)):
        step()
    fence()
    _lib.profile_enable(True)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    fence()
    t_start = datetime.datetime.now()
    ev0.record()
    for _ in range(a.steps):
        root = step()
    ev1.record()
    fence()
    t_end = datetime.datetime.now()
    ms = ev0.elapsed_time(ev1)
    prof = _lib.profile_read()
    _lib.profile_enable(False)
    clocks = sampler.stop(t_start, t_end) if rank == 0 else None
    root_hex = bytes(root.cpu().tolist()).hex()

    # end to end: pinned host input -> H2D -> commit -> D2H root, all inside the timed region; beside it
    # the bare copy of the same pinned rows in the same slices (what the host and PCIe path allow)
    e2e_ms, h2d_ms, host = 0.0, 0.0, None
    if not a.no_e2e:
        host = torch.empty((rows, k), dtype=torch.uint64).pin_memory()
        host.copy_(msg)
        torch.cuda.synchronize()
        for _ in range(2):
            com.commit_host(host)
        fence()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        for _ in range(a.steps):
            rb = com.commit_host(host)
        t1.record()
        fence()
        e2e_ms = t0.elapsed_time(t1)
        assert rb.hex() == root_hex, "host-path root differs from the device-path root"
        com.copy_only(host)
        fence()
        t0.record()
        for _ in range(a.steps):
            com.copy_only(host)
        t1.record()
        fence()
        h2d_ms = t0.elapsed_time(t1)
    h2d_bytes, d2h_bytes = com.h2d_bytes, com.d2h_bytes
    del com, host
    torch.cuda.empty_cache()

    # ---- ONE tree over `rows` rows split over the ranks --------------------------------------------
    sharded, payload = {}, {}
    if not a.no_sharded:
        from verinf_b200 import cuda_primitives as cp
        backend = D.CudaBackend(k, n)
        # small case first: sharded root == single-GPU root of the concatenated rows (checked on every rank)
        s_rows, s_k = 1024, 1 << 12
        small = gen_rows(torch, dev, 0, s_rows, s_k, s_rows, seed0=SEED + 100)
        r0, r1 = D.split_rows(s_rows, world)[rank]
        s_root, _, _ = D.commit_rows_sharded(small[r0:r1].contiguous(), s_rows, D.CudaBackend(s_k, 4 * s_k))
        want, _, _ = cp.commit_rows(small, s_k, 4 * s_k)
        small_ok = all_agree(torch, dist, world, dev, bool(torch.equal(s_root, want)))
        assert small_ok, "sharded commit root differs from the single-GPU root (1024 x 2^12 case)"
        del small
        r0, r1 = D.split_rows(rows, world)[rank]
        mine = msg[r0:r1].contiguous() if world == 1 else gen_rows(torch, dev, r0, r1, k, rows)
        for _ in range(2):
            D.commit_rows_sharded(mine, rows, backend)
        fence()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        for _ in range(a.steps):
            sh_root, _, sh_codes = D.commit_rows_sharded(mine, rows, backend)
        t1.record()
        fence()
        sh_hex = bytes(sh_root.cpu().tolist()).hex()
        if world == 1:
            assert sh_hex == root_hex, "sharded path at one rank must reproduce the headline root"
        sharded["commit_ms"] = t0.elapsed_time(t1) / a.steps
        sharded["commit_root"] = sh_hex
        del mine, sh_codes
        torch.cuda.empty_cache()

        # ---- sharded sumcheck: 3 tables x 2^24, coins drawn before it starts -------------------------
        from verinf_b200 import layergkr_gpu as lg
        tabs = sumcheck_tables(torch, dev)
        coins = sumcheck_coins()
        terms = [(1, [0, 1, 2])]
        shard = D.shard_table(tabs, rank, world)
        mk = lambda t: lg.SumcheckProblem(t.contiguous(), terms)
        sc_ms = []
        for it in range(2 + min(a.steps, 5)):
            prob = lg.SumcheckProblem(shard.clone(), terms)
            fence()
            t0.record()
            claim, polys, _ = D.prove_terms_sharded(prob, mk, None, SC_LOG, dev, coins=coins)
            t1.record()
            torch.cuda.synchronize()
            if it >= 2:
                sc_ms.append(t0.elapsed_time(t1))
        ys = [[y for _, y in rp] for rp in polys]
        if world > 1:      # rank 0 holds the whole tables: the unsharded prover must give the same transcript
            same = True
            if rank == 0:
                full = lg.SumcheckProblem(tabs.clone(), terms)
                same = full.run(coins) == ys
            assert all_agree(torch, dist, world, dev, same), "sharded sumcheck transcript differs from the unsharded one"
        sharded["sumcheck_ms"] = min(sc_ms)
        sharded["sumcheck_digest"] = hashlib.sha256(repr((claim, ys)).encode()).hexdigest()[:16]
        if world == 1 and not a.no_cpu:
            payload["sumcheck"] = {"tables": tabs.view(torch.int64).cpu().numpy().view("uint64"), "coins": coins,
                                   "claim": claim, "polys": ys}
        del tabs, shard, prob
        torch.cuda.empty_cache()

    t = torch.tensor([ms, e2e_ms, h2d_ms, sharded.get("commit_ms", 0.0), sharded.get("sumcheck_ms", 0.0)],
                     dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms, e2e_ms, h2d_ms, sh_commit_ms, sh_sc_ms = (float(x) for x in t)

    # ---- second half of the metric, on rank 0 (the other ranks wait at the barrier below) ----------
    extra = {}
    check = world == 1 and not a.no_cpu
    if rank == 0 and not a.no_secondary:
        from verinf_b200 import workloads
        kq = [workloads.kquant_fused_encode(dev, q, check_rows=[0, -1] + [997 * i % 5504 for i in range(1, 17)]
                                            if check else None) for q in ("Q4_K", "Q6_K")]
        payload["kquant"] = [dict(r.pop("_check"), qtype=r["qtype"]) for r in kq if "_check" in r]
        extra["kquant_fused_encode"] = kq
        ly = workloads.layer7b_commit_sumcheck(dev, with_check=check)
        if "_check" in ly:
            payload["layer7b"] = ly.pop("_check")
        extra["layer7b"] = ly
        torch.cuda.empty_cache()
    if rank == 0 and a.extra:
        from verinf_b200 import workloads
        extra["field_matmul"] = workloads.field_matmul(dev)
        extra["fold_products"] = workloads.fold_products(dev)
        if world == 1:          # one GPU only: the reference's extension takes a minute or two to JIT-build
            extra["reference_cuda"] = reference_cuda_leg()
    if a.extra:
        # MoE variant: 128 experts x (5120 x 8192) int8, 16 per GPU at 8 GPUs, one commitment per expert,
        # roots gathered; with fewer ranks every rank still commits 16 experts (rank r: 16r .. 16r+15)
        from verinf_b200 import workloads
        mo = workloads.moe_expert_commits(dev, list(range(16 * rank, 16 * rank + 16)), prefix_check=check)
        if "_check" in mo:
            payload["moe"] = mo.pop("_check")
        all_roots = [None] * world
        if world > 1:
            dist.all_gather_object(all_roots, mo["roots"])
        else:
            all_roots = [mo["roots"]]
        tt = torch.tensor([mo["seconds"]], dtype=torch.float64, device=dev)
        if world > 1:
            dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        flat = [r for rs in all_roots for r in rs]
        extra["moe_expert_commits"] = {
            "experts_committed": len(flat), "experts_per_gpu": 16, "of_experts": 128,
            "expert_shape": [5120, 8192], "rows_per_gpu": mo["rows"], "seconds": float(tt[0]),
            "codeword_gb_per_gpu": mo["codeword_gb"], "first_root": flat[0].hex(),
            "roots_sha256": hashlib.sha256(b"".join(flat)).hexdigest()}
    if world > 1:
        dist.barrier()

    if rank == 0:
        elems = world * rows * n
        hbm_peak, peak_src = peaks()
        # dominant kernel = the tag with the largest share of device time in the timed region
        total_prof = sum(v[0] for v in prof.values()) or 1.0
        dom = max(prof.items(), key=lambda kv: kv[1][0])
        per_row = {"encode_pass1": 8 * (k + k), "encode_mid": 8 * (k + n), "encode_pass3": 8 * (n + n),
                   "hash_columns": 8 * n}
        # DRAM bytes per message row from ncu captures of these kernels (dram read + write of one launch /
        # rows of that launch), valid for this geometry only; scaled to an average launch
        ncu_per_row = {"encode_pass1": 0.938e6, "encode_mid": 2.484e6, "encode_pass3": 4.074e6,
                       "hash_columns": 2.193e6} if (a.log_k, a.blowup) == (16, 4) else {}
        launches = sum(v[1] for v in prof.values())
        bytes_per_step = rows * per_row.get(dom[0], 0)
        dom_ms_per_step = dom[1][0] / a.steps
        achieved = bytes_per_step / (dom_ms_per_step * 1e-3) / 1e9 if dom_ms_per_step else 0.0
        enc_ms = sum(prof.get(t_, (0, 0))[0] for t_ in ("encode_pass1", "encode_mid", "encode_pass3")) / a.steps
        # integer roofline of the encode: issue slots of its arithmetic, measured with the integer-pipe microbenchmark
        # (a radix-16 butterfly 43 per element, 10.75 per radix-2 element-stage; a multiply 32), against 148 SMs x 4
        # schedulers x 32 lanes per clock at the SM clock sampled during the run.  The coset twist is a multiply of
        # its own only for blow-up factors other than 2 and 4.
        stages_per_row = (1 + a.blowup) * k * a.log_k
        muls_per_row = (1 + a.blowup) * k * 3 + a.blowup * k + k
        issue_muls = muls_per_row - (a.blowup * k if a.blowup in (2, 4) else 0)
        sm_hz = ((clocks or {}).get("sm_mhz") or 1965.0) * 1e6
        issue_floor_ms = rows * (stages_per_row * 10.75 + issue_muls * 32) / (148 * 128 * sm_hz) * 1e3
        # the two-term roofline the path's target is stated in: the slower of the bytes at the HBM peak and the
        # full modular multiplies at the measured multiply rate (855 G/s at 1965 MHz, integer-pipe microbenchmark);
        # butterflies, which are most of the work, are in neither term
        modmul_ms = rows * muls_per_row / (855e9 * sm_hz / 1965e6) * 1e3
        bytes_ms = rows * 8 * (k + n) / (hbm_peak * 1e9) * 1e3
        line = {
            "metric": METRIC, "value": elems * a.steps / (ms * 1e-3), "unit": UNIT, "n_gpus": world,
            "steps": a.steps, "warmup": max(a.warmup, 3), "ms_per_step": ms / a.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u64",
            "data": "synthetic",
            "config": {"workload": workload_name(a), "rows_per_gpu": rows, "K": k, "N": n,
                       "l2_policy": "inputs (2 GiB) and outputs (8 GiB) exceed L2; no flush needed",
                       "numa_bound": numa_bound,
                       "root": root_hex},
            # the fraction is of the HBM roofline (algorithmic bytes / time against the measured copy peak), as
            # the metric asks; the kernel's limiter is integer issue, whose floor is `int_roofline`
            "roofline": {"bound": "hbm", "limiter": "integer issue (see int_roofline)", "kernel": dom[0],
                         "achieved": achieved, "peak": hbm_peak,
                         "unit": "GB/s", "frac": achieved / hbm_peak, "peak_source": peak_src,
                         "traffic": (ncu_per_row[dom[0]] * rows * a.steps / dom[1][1]) if dom[0] in ncu_per_row else None,
                         "launches_per_step": dom[1][1] / a.steps,
                         "ms_per_launch": dom[1][0] / dom[1][1],
                         "algorithmic_bytes_per_step": bytes_per_step,
                         "share_of_device_time": dom[1][0] / total_prof},
            "kernels": {t_: {"ms_per_step": v[0] / a.steps, "launches_per_step": v[1] / a.steps,
                             "share": v[0] / total_prof,
                             "gbs": rows * per_row.get(t_, 0) / (v[0] / a.steps * 1e-3) / 1e9 if v[0] else None}
                        for t_, v in prof.items()},
            "encode_only": {"ms_per_step": enc_ms,
                            "gbs_algorithmic": rows * 8 * (k + n) / (enc_ms * 1e-3) / 1e9 if enc_ms else None,
                            "frac_of_hbm": rows * 8 * (k + n) / (enc_ms * 1e-3) / 1e9 / hbm_peak if enc_ms else None},
            "int_roofline": {"bound": "integer issue slots (128 lanes/clk/SM)", "encode_floor_ms": issue_floor_ms,
                             "bytes_or_modmul_floor_ms": max(modmul_ms, bytes_ms), "modmul_floor_ms": modmul_ms,
                             "frac_of_bytes_or_modmul_floor": max(modmul_ms, bytes_ms) / enc_ms if enc_ms else None,
                             "encode_ms": enc_ms, "frac": issue_floor_ms / enc_ms if enc_ms else None},
            "gpu_launches": launches,
            "clocks": clocks,
        }
        if e2e_ms:
            line["e2e"] = {"value": elems * a.steps / (e2e_ms * 1e-3), "unit": UNIT,
                           "h2d_bytes_per_step": h2d_bytes, "d2h_bytes_per_step": d2h_bytes,
                           "ms_per_step": e2e_ms / a.steps, "h2d_only_ms": h2d_ms / a.steps,
                           "h2d_only_gbs_per_gpu": h2d_bytes / (h2d_ms / a.steps * 1e-3) / 1e9 if h2d_ms else None}
        if sharded:
            sc_bytes = 4 * 3 * (1 << SC_LOG) * 8
            line["sharded_commit"] = {
                "what": f"ONE tree over {rows} rows, {rows // world} per rank, sub-tree values all-gathered",
                "ms": sh_commit_ms, "elems_per_s": rows * n / (sh_commit_ms * 1e-3), "root": sharded["commit_root"],
                "small_case_root_equals_single_gpu": True}
            line["sharded_sumcheck"] = {
                "what": f"degree-3 product of three 2^{SC_LOG} tables, {SC_LOG} rounds, entries i mod {world} per rank, "
                        "coins from Transcript(b'bench/sumcheck'); partial sums all-reduced as 32-bit limbs",
                "ms": sh_sc_ms, "transcript_digest": sharded["sumcheck_digest"],
                "roofline": {"bound": "hbm", "algorithmic_bytes": sc_bytes,
                             "achieved": sc_bytes / (sh_sc_ms * 1e-3) / 1e9 / world, "peak": hbm_peak,
                             "unit": "GB/s per GPU", "frac": sc_bytes / (sh_sc_ms * 1e-3) / 1e9 / world / hbm_peak}}
        line.update(extra)
        if "layer7b" in extra:
            line["layer7b_commit_plus_sumcheck_s"] = extra["layer7b"]["commit_plus_sumcheck_s"]
        if check:
            line.update(cpu_self_check(a, torch, msg, root_hex, k, n, payload))
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


def reference_cuda_leg():
    """The reference's own CUDA kernels beside this library on the same GPU (second, independent
    witness and same-box number): tests/reference_runner.py runs `encode_messages`,
    `hash_columns_streamed`, `merkle_build_blake3` and a batched NTT at the geometry the reference's
    authors validated (ELL=8192, K=16384, N=65536, 1024 rows) once on the reference's JIT-built
    extension and once on this library, from the staged tree baseline/_ref; digests must agree."""
    runner = ROOT / "tests" / "reference_runner.py"
    if not (ROOT / "baseline" / "_ref" / "prover" / "core.py").exists():
        return {"unavailable": "baseline/_ref not staged (python baseline/stage_reference.py)"}
    env = dict(os.environ)
    env.setdefault("TORCH_EXTENSIONS_DIR", str(ROOT / "build" / "torch_extensions"))
    res = {}
    for backend in ("reference", "shim"):
        p = subprocess.run([sys.executable, str(runner), "--backend", backend, "--job", "kernels"], capture_output=True,
                           text=True, timeout=1500, env=env, cwd=str(ROOT))
        lines = [ln for ln in p.stdout.splitlines() if ln.startswith("{")]
        res[backend] = json.loads(lines[-1]) if lines else {"error": p.stderr[-500:]}
        if "error" in res[backend]:
            return {"unavailable": f"{backend} run failed: " + res[backend]["error"][-300:]}
    ref, ours = res["reference"], res["shim"]
    keys = ("polys_sha256", "codes_sha256", "leaves_sha256", "root", "ntt64x65536_sha256")
    return {"geometry": {"rows": ref["rows"], "ELL": ref["ELL"], "K": ref["K"], "N": ref["N"]},
            "bit_identical": all(ref[k_] == ours[k_] for k_ in keys),
            "encode_ms": ref["encode_ms"], "hash_ms": ref["hash_ms"], "merkle_ms": ref["merkle_ms"],
            "ntt_64x65536_ms": ref["ntt64x65536_x3_ms"],
            "ours_encode_ms": ours["encode_ms"], "ours_hash_ms": ours["hash_ms"], "ours_merkle_ms": ours["merkle_ms"],
            "ours_ntt_64x65536_ms": ours["ntt64x65536_x3_ms"]}


def time_sumcheck(torch, dev):
    """Degree-3 product of three 2^24 tables, 24 rounds, coins pre-drawn from the seeded transcript (all
    rounds queued + one D2H; the claim is the first round's g(0) + g(1))."""
    from verinf_b200 import layergkr_gpu as lg
    tabs = sumcheck_tables(torch, dev)
    coins = sumcheck_coins()
    best = None
    for _ in range(3):
        t = tabs.clone()
        prob = lg.SumcheckProblem(t, [(1, [0, 1, 2])])
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ys = prob.run(coins)                       # all rounds queued; g(1) of later rounds derived on the host
        claim = (ys[0][0] + ys[0][1]) % P          # the sum over the hypercube is g_0(0) + g_0(1)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
        best = dt if best is None else min(best, dt)
    nbytes = 4 * 3 * (1 << 24) * 8
    return {"ms": best * 1e3, "algorithmic_gbs": nbytes / best / 1e9, "claim": claim}


def build_int_pipes():
    """Compiles the integer-pipe / field-primitive microbenchmark (bench_int_pipes.cu) for sm_100a."""
    from verinf_b200.build import _nvcc
    out = ROOT / "build" / "int_pipes"
    src = ROOT / "bench_int_pipes.cu"
    out.parent.mkdir(exist_ok=True)
    deps = [src] + sorted((ROOT / "verinf_b200" / "csrc").glob("*.cuh"))
    if not out.exists() or out.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        env = {k_: v for k_, v in os.environ.items() if k_ not in ("CC", "CXX")}
        subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
                               "--expt-relaxed-constexpr", "-I", str(ROOT), "-o", str(out), str(src)], env=env)
    return out


def run_micro(a):
    if a.micro == "int_pipes":
        sys.exit(subprocess.call([str(build_int_pipes())]))
    import torch
    from verinf_b200 import workloads
    dev = torch.device("cuda:0")
    torch.cuda.set_device(dev)
    if a.micro == "matmul":
        out = workloads.field_matmul(dev, 1024, 2048, 2048)
    elif a.micro == "fold":
        out = workloads.fold_products(dev)
    else:
        out = time_sumcheck(torch, dev)
    print(json.dumps({"micro": a.micro, **out}))


if __name__ == "__main__":
    args = parse()
    if args.micro:
        run_micro(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_native(args)
