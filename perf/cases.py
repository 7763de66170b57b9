"""Timed cases of the PAR2 recovery engine: what a program has it do, over its real range.

Every case runs through the package's public entry points: the GfProc backend
(host slices in, host recovery slices out), the device-level contraction
par2cuda_muladd, the resident job (with and without hashes), the job stream,
the batch runner and the IFSC hashes.  The sizes are those of the benchmark
workloads and of the uneven job mix (10..5000 input slices of 64 KiB..8 MiB,
recovery 1..30 % of the inputs), odd ones included.  Slice data is uniform
random, as archives and media are.  Every output is a whole number or a byte.
"""
import math

import numpy as np
import torch

from parpar_gb300 import _lib
from parpar_gb300.batch import BatchRunner, JobSpec
from parpar_gb300.gfproc import GfProc
from parpar_gb300.job import ResidentJob
from parpar_gb300.layout import file_lengths
from parpar_gb300.stream import JobStream

KIB, MIB = 1024, 1024 * 1024


def listed():
    return [
        # a small set through the backend as the addon drives it: pageable buffers, defaults
        {"name": "gfproc_small", "kind": "gfproc", "n": 16, "s": 64 * KIB, "r": 4, "method": "auto", "batch": 0,
         "pinned": False},
        # an ordinary set through the backend in several accumulating batches, pinned buffers
        {"name": "gfproc_batches", "kind": "gfproc", "n": 300, "s": MIB, "r": 30, "method": "tensor_fp4", "batch": 128,
         "pinned": True},
        # the smallest jobs of a mix: launch-bound
        {"name": "muladd_tiny", "kind": "muladd", "n": 10, "s": 64 * KIB, "r": 1, "method": "auto", "acc": False},
        # the default method on resident slices, added onto earlier recovery data
        {"name": "muladd_auto_acc", "kind": "muladd", "n": 500, "s": 512 * KIB + 20, "r": 50, "method": "auto", "acc": True},
        # 100 slices of 1 MiB, 10 recovery slices: the plain create
        {"name": "muladd_plain", "kind": "muladd", "n": 100, "s": MIB, "r": 10, "method": "tensor_fp4", "acc": False},
        # a mid job of the mix: odd counts, a slice size that is no multiple of any tile
        {"name": "muladd_ragged", "kind": "muladd", "n": 777, "s": 1400012, "r": 133, "method": "tensor_fp4", "acc": False},
        # 4 GiB of slices, 10 % recovery: checksums, contraction, verification
        {"name": "job_bandwidth", "kind": "job", "n": 2000, "s": 2 * MIB, "r": 200, "files": 40, "method": "tensor_fp4",
         "hashes": False},
        # as many recovery slices as inputs: the largest contraction
        {"name": "job_dense", "kind": "job", "n": 4096, "s": 256 * KIB, "r": 4096, "files": 1, "method": "tensor_fp4",
         "hashes": False},
        # a whole create on the device: IFSC, file MD5s and recovery packet MD5s too; the slice size
        # is what dividing files into a given number of slices gives, a multiple of 4
        {"name": "job_hashes", "kind": "job", "n": 200, "s": 300012, "r": 20, "files": 12, "method": "comb",
         "hashes": True},
        # several creates in flight, from and to pinned host buffers
        {"name": "stream_host", "kind": "stream", "n": 160, "s": 256 * KIB, "r": 24, "files": 16, "jobs": 8},
        # small jobs of uneven sizes in one captured graph
        {"name": "batch_mix", "kind": "batch", "jobs": 24, "nmax": 600, "smax": MIB},
        # per-slice MD5 + CRC32 alone
        {"name": "ifsc", "kind": "ifsc", "n": 2000, "s": 256 * KIB + 44},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["muladd", "muladd", "muladd", "muladd", "job", "job", "gfproc", "stream", "batch", "ifsc"])
    if kind == "ifsc":
        return {"kind": kind, "n": _logint(rng, 10, 5000), "s": 4 * _logint(rng, 4 * KIB, 128 * KIB)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(8, 32), "nmax": _logint(rng, 100, 600), "smax": 4 * _logint(rng, 32 * KIB, MIB // 4)}
    if kind == "stream":
        return {"kind": kind, "n": _logint(rng, 40, 160), "s": 64 * _logint(rng, KIB, 4 * KIB), "r": rng.randint(4, 40),
                "files": rng.randint(4, 16), "jobs": rng.choice([4, 8])}
    n = _logint(rng, 10, 2500)
    r = max(1, int(round(rng.uniform(0.01, 0.30) * n)))
    s = 4 * _logint(rng, 16 * KIB, 2 * MIB)
    if kind == "gfproc":
        n = min(n, 400)
        r = min(r, 60)
        s = min(s, 256 * MIB // n // 4 * 4)
        return {"kind": kind, "n": n, "s": s, "r": r, "method": rng.choice(["auto", "tensor_fp4"]), "batch": rng.choice([0, 64]),
                "pinned": rng.random() < 0.5}
    s = max(256, min(s, 4 * 1024 * MIB // n // 4 * 4))
    if kind == "job":
        hashes = rng.random() < 0.3
        if hashes:
            n = min(n, 300)
            files = min(n, 12)
            r, s = min(r, 60), min(s, 8 * MIB * files // (2 * n) // 4 * 4)   # the longest file about 8 MiB
        else:
            files = min(n, rng.randint(1, 40))
        return {"kind": kind, "n": n, "s": s, "r": r, "files": files,
                "method": rng.choice(["comb", "tensor_fp4", "tensor_fp4"]), "hashes": hashes}
    return {"kind": kind, "n": n, "s": s, "r": r, "method": rng.choice(["auto", "tensor_fp4", "tensor_fp4"]),
            "acc": rng.random() < 0.3}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _fill(t, g):
    """Uniform random bytes into a device tensor."""
    t.view(torch.int32).random_(-(1 << 31), (1 << 31) - 1, generator=g)


def _batch_specs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for j in range(case["jobs"]):
        n = int(round(math.exp(rng.uniform(math.log(10), math.log(case["nmax"])))))
        s = int(rng.integers(64 * KIB // 4, case["smax"] // 4 + 1)) * 4
        r = max(1, int(round(rng.uniform(0.01, 0.30) * n)))
        out.append((n, s, r, j))
    return out


def prepare(case, seed):
    L = _lib.load()
    kind = case["kind"]
    g = _gen(seed)
    st = {"kind": kind, "case": case, "L": L}
    if kind == "muladd":
        n, s, r = case["n"], case["s"], case["r"]
        pitch = L.par2cuda_row_pitch_bytes(s)
        st["pw"] = pw = pitch // 2
        st["nw"] = nw = ((s + 7) // 8 * 8 + 8) // 2
        st["d_in"] = torch.zeros((n, pw), dtype=torch.int16, device="cuda")
        _fill(st["d_in"], g)
        st["d_rec"] = torch.zeros((r, pw), dtype=torch.int16, device="cuda")
        if case["acc"]:
            _fill(st["d_rec"], g)
        nums = torch.arange(n, dtype=torch.int16, device="cuda")
        exps = torch.arange(r, dtype=torch.int16, device="cuda")
        st["d_coeff"] = torch.empty((r, n), dtype=torch.int16, device="cuda")
        _lib.check(L.par2cuda_par2_coeffs(nums.data_ptr(), n, exps.data_ptr(), r, st["d_coeff"].data_ptr(), None), "coeffs")
        st["method"] = _lib.METHOD_NAMES[case["method"]]
        sb = L.par2cuda_muladd_scratch_bytes(r, n)
        if case["method"] == "tensor_fp4":
            sb = L.par2cuda_tensor_fp4_scratch_bytes(r, n, nw)
        st["d_scratch"] = torch.empty(max(sb, 256), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
    elif kind == "gfproc":
        n, s, r = case["n"], case["s"], case["r"]
        pitch = (s + 3) // 4 * 4
        d = torch.empty((n, pitch), dtype=torch.uint8, device="cuda")
        _fill(d, g)
        st["host_in"] = torch.empty((n, pitch), dtype=torch.uint8, pin_memory=case["pinned"])
        st["host_in"].copy_(d)
        st["host_out"] = torch.zeros((r, s), dtype=torch.uint8, pin_memory=case["pinned"])
        st["ins"] = [st["host_in"][i, :s] for i in range(n)]
        st["outs"] = [st["host_out"][i] for i in range(r)]
        st["proc"] = GfProc(s, method=case["method"], input_batchsize=case["batch"])
        st["proc"].set_recovery_slices(range(r))
    elif kind == "job":
        lens = file_lengths(case["n"], case["files"], case["s"], seed)
        job = ResidentJob(case["s"], lens, list(range(case["r"])), method=_lib.METHOD_NAMES[case["method"]])
        _fill(job.d_in, g)
        st["job"] = job
        torch.cuda.synchronize()
    elif kind == "stream":
        lens = file_lengths(case["n"], case["files"], case["s"], seed)
        js = JobStream(case["s"], lens, list(range(case["r"])), slots=8, group=4, method=_lib.METHOD_TENSOR_FP4)
        d = torch.empty((case["n"], case["s"]), dtype=torch.uint8, device="cuda")
        st["host_in"] = []
        for _ in range(2):
            _fill(d, g)
            h = torch.empty((case["n"], case["s"]), dtype=torch.uint8, pin_memory=True)
            h.copy_(d)
            st["host_in"].append(h)
        st["host_out"] = js.host_out_buffers(case["jobs"])
        st["stream"] = js
    elif kind == "batch":
        # fixed sizes (they are the case), the slices' bytes from the seed
        specs = [JobSpec(n, s, r, int(seed) * 1000 + j, list(range(r))) for n, s, r, j in _batch_specs(case, 4)]
        runner = BatchRunner(specs, shape_of=lambda R: 5 if R > 8 else 1, method_of=lambda R: "tensor_fp4", mode="grid")
        runner.capture()
        st["runner"] = runner
        torch.cuda.synchronize()
    else:
        n, s = case["n"], case["s"]
        st["pitch"] = pitch = L.par2cuda_row_pitch_bytes(s)
        st["d_in"] = torch.empty((n, pitch), dtype=torch.uint8, device="cuda")
        _fill(st["d_in"], g)
        st["d_ifsc"] = torch.empty((n, 20), dtype=torch.uint8, device="cuda")
        # every tenth slice ends a file
        lens = np.full(n, s, dtype=np.int32)
        lens[::10] = np.random.default_rng(seed).integers(1, s + 1, size=len(lens[::10]))
        st["d_lens"] = torch.from_numpy(lens).cuda()
    return st


def run(st):
    kind, case, L = st["kind"], st["case"], st["L"]
    cur = torch.cuda.current_stream().cuda_stream
    if kind == "muladd":
        pw, sc = st["pw"], st["d_scratch"]
        _lib.check(L.par2cuda_muladd(st["d_in"].data_ptr(), pw, case["n"], st["d_coeff"].data_ptr(), st["d_rec"].data_ptr(), pw,
                                     case["r"], st["nw"], int(case["acc"]), st["method"], sc.data_ptr(), sc.numel(), cur), "muladd")
        return st["d_rec"][:, : st["nw"]]
    if kind == "gfproc":
        p = st["proc"]
        for i, buf in enumerate(st["ins"]):
            p.add_sync(i, buf)
        p.end_sync()
        valid = []
        for r, out in enumerate(st["outs"]):
            p.get(r, out, lambda idx, ok, _: valid.append((idx, ok)))
        p.sync()
        return {"rec": st["host_out"], "valid": np.array([int(ok) for _, ok in sorted(valid)])}
    if kind == "job":
        job = st["job"]
        job.run(hashes=case["hashes"])
        out = {"rec": job.d_rec[:, : job.row_words], "valid": job.d_flags}
        if case["hashes"]:
            out["packets"] = np.frombuffer(b"".join(job.recovery_packet_md5s(bytes(range(16)))), dtype=np.uint8)
            out["ifsc"], out["fmd5"] = job.d_ifsc, job.d_fmd5
        return out
    if kind == "stream":
        st["stream"].clear_records()
        st["stream"].run(case["jobs"], host_in=st["host_in"], host_out=st["host_out"])
        torch.cuda.current_stream().synchronize()   # the results are read on the host
        return {"job%d" % k: list(o) for k, o in enumerate(st["host_out"])}
    if kind == "batch":
        st["runner"].run_batched()
        return [x for b in st["runner"].bufs for x in (b.d_rec.view(torch.uint8)[:, : b.spec.S], b.d_flags)]
    _lib.check(L.par2cuda_slice_hash(st["d_in"].data_ptr(), st["pitch"], case["n"], st["d_lens"].data_ptr(), case["s"],
                                     st["d_ifsc"].data_ptr(), cur), "slice_hash")
    return st["d_ifsc"]


def exact(case, seed):
    # field arithmetic and hashes: every output is a whole number or a byte
    return None


def work(case):
    """Bytes: each input read once and each output written once.  Flops: two
    three-input XORs per 16-bit word multiply-add; hashes count none."""
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_specs(case, 4)
        return {"bytes": sum((n + r) * s for n, s, r, _ in specs), "flops": sum(n * r * s // 2 * 2 for n, s, r, _ in specs)}
    n, s = case["n"], case["s"]
    if kind == "ifsc":
        return {"bytes": n * s + 20 * n, "flops": 0}
    r = case["r"]
    jobs = case.get("jobs", 1)
    return {"bytes": jobs * (n + r) * s + 2 * n * r, "flops": jobs * n * r * (s // 2) * 2}
