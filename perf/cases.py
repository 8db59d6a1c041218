"""Performance cases of the framework: what its users run, through the public entry points.

A case is a dict of plain values; `kind` names the path:

  ntt1d     single-modulus negacyclic NTT, forward and inverse (cbs_fnwt_1d_*, cbs_inwt_1d_*)
  ntt2d     multi-prime NTT of RNS polynomials, forward and inverse (cbs_rns_ntt_batched)
  keyswitch hybrid key switch of a batch of ciphertexts (cbs_rns_keyswitch_inplace)
  ckks      one CKKS multiply + relinearize + rescale, or one rotation
  gate      a batch of gate bootstraps (cbs_gate_eval_batch_device)
  ragged    requests of uneven size over two gate parameter sets, one launch per set
  aes       AES-128 CTR transciphering from host buffers, then decryption by the key owner
  cbs       circuit bootstrapping with an exact blind rotation, RGSW rows out
  tcb       torus circuit bootstrapping with private functional key switching

Integer outputs (residues, torus words, RGSW rows, decrypted bits) are compared exactly.  Where a
path's ciphertexts carry FP64 rounding in their noise (aes, tcb, split FP32 gates), two correct
implementations give different, equally random words, so the pass ends with the decryption
that gives them a meaning: plaintext bits, or for tcb the phases of all RGSW rows.
"""
import importlib.util
import math
import os
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
# untuned defaults: no tuning cache of the machine decides what a case launches
os.environ["CBS_TUNE_CACHE"] = os.path.join(tempfile.gettempdir(), "cbs_perf_no_tune_cache.json")

_held = {}  # plans, keys and contexts a program keeps for its lifetime, by configuration


def _pkg():
    name = "cbs_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            name, ROOT / "gpu-circuitbootstrapping-aestransciphering_b200" / "__init__.py")
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def _keep(key, make):
    if key not in _held:
        _held[key] = make()
    return _held[key]


# ---------------------------------------------------------------------------- the cases

def listed():
    return [
        # one RGSW ciphertext's polynomials: the smallest transform call, bound by its launch
        {"name": "ntt1d_16", "kind": "ntt1d", "logn": 11, "polys": 16},
        # 8 two-polynomial ciphertexts at the CKKS ring and depth of the Phantom workloads
        {"name": "ntt2d_2p16x24x16", "kind": "ntt2d", "logn": 16, "bits": 50, "limbs": 24, "polys": 16},
        # key switches of a batch, the same ring with two special primes (12 digits)
        {"name": "keyswitch_2p16_24p2_x4", "kind": "keyswitch", "logn": 16, "bits": 50, "size_q": 24, "size_p": 2,
         "level": 24, "count": 4},
        # one ciphertext product at a middle ring: a few MB of work in many launches
        {"name": "ckks_mul_2p15_12p2", "kind": "ckks", "op": "mul", "logn": 15, "bits": 50, "size_q": 12, "size_p": 2,
         "level": 12},
        # one rotation with 59-bit primes, below the top level (a ragged last digit): integer kernels
        {"name": "ckks_rot_2p14_9p2_59b", "kind": "ckks", "op": "rotate", "logn": 14, "bits": 59, "size_q": 9,
         "size_p": 2, "level": 7},
        # a small circuit layer of independent gates: fewer ciphertexts than SMs
        {"name": "gate_64", "kind": "gate", "mode": "fp64", "mb": 2, "count": 64},
        # a serving mix over both gate parameter sets, uneven requests
        {"name": "ragged_1731", "kind": "ragged", "mode": "fp64", "mb": 2, "small": "301,1,517,64", "large": "129,33,686"},
        # the same gates with split-FP32 products, one full wave
        {"name": "gate_f32split_592", "kind": "gate", "mode": "fp32-split", "mb": 1, "count": 592},
        # AES-128: the latency of one block, and a batch of an odd number of blocks
        {"name": "aes_1", "kind": "aes", "blocks": 1},
        {"name": "aes_13", "kind": "aes", "blocks": 13},
        # bits to RGSW with exact products, for callers that run their own CMux trees
        {"name": "cbs_split_200", "kind": "cbs", "params": "2x18", "backend": "split", "mb": 2, "count": 200},
        # bits to torus RGSW through PFKS
        {"name": "tcb_48", "kind": "tcb", "mb": 2, "count": 48},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ntt1d", "ntt2d", "ntt2d", "keyswitch", "keyswitch", "ckks", "ckks", "gate", "gate", "gate",
                       "ragged", "aes", "aes", "cbs", "cbs", "tcb"])
    if kind == "ntt1d":
        return {"kind": kind, "logn": rng.choice([10, 11, 12]), "polys": _log_int(rng, 1, 8192)}
    if kind == "ntt2d":
        logn = rng.randint(12, 17)
        limbs = rng.randint(1, 30)
        return {"kind": kind, "logn": logn, "bits": rng.choice([40, 50, 50, 59]), "limbs": limbs,
                "polys": _log_int(rng, 1, max(2, min(256, (1 << 25) // (limbs << logn))))}
    if kind == "keyswitch":
        size_q = rng.randint(3, 24)
        logn = rng.randint(12, 16)
        return {"kind": kind, "logn": logn, "bits": rng.choice([45, 50, 50, 59]), "size_q": size_q,
                "size_p": min(size_q, rng.choice([1, 2, 2, 3, 8])), "level": rng.randint(max(2, size_q // 2), size_q),
                "count": _log_int(rng, 1, 6 if logn == 16 else 12)}
    if kind == "ckks":
        size_q = rng.randint(3, 20)
        return {"kind": kind, "op": rng.choice(["mul", "rotate"]), "logn": rng.randint(12, 16),
                "bits": rng.choice([45, 50, 50, 59]), "size_q": size_q, "size_p": min(size_q, rng.choice([1, 2, 3, 4])),
                "level": rng.randint(2, size_q)}
    if kind == "gate":
        mode = rng.choice(["fp64", "fp64", "fp64", "fp32-split"])
        return {"kind": kind, "mode": mode, "mb": rng.choice([1, 2, 2, 3]) if mode == "fp64" else 1,
                "count": _log_int(rng, 1, 4736)}
    if kind == "ragged":
        sizes = [str(_log_int(rng, 1, 900)) for _ in range(rng.randint(2, 6))]
        k = rng.randint(1, len(sizes) - 1)
        return {"kind": kind, "mode": "fp64", "mb": rng.choice([1, 2]), "small": ",".join(sizes[:k]),
                "large": ",".join(sizes[k:])}
    if kind == "aes":
        return {"kind": kind, "blocks": rng.randint(1, 12)}
    if kind == "cbs":
        backend = rng.choice(["split", "split", "ntt"])
        return {"kind": kind, "params": rng.choice(["2x18", "3x12"]), "backend": backend,
                "mb": rng.choice([1, 2]) if backend == "split" else 1, "count": _log_int(rng, 1, 300)}
    return {"kind": kind, "mb": rng.choice([1, 2]), "count": _log_int(rng, 1, 200)}


# ---------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _residues(g, lead, mods, n):
    """Uniform residues [*lead][len(mods)][n]: what NTT-domain ciphertexts and keys hold."""
    m = torch.from_numpy(np.asarray(mods, np.uint64).view(np.int64)).cuda().view(-1, 1)
    t = torch.randint(0, 2 ** 62, (*lead, len(mods), n), dtype=torch.int64, device="cuda", generator=g)
    return torch.remainder(t, m).contiguous()


def _dev32(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


class _View:
    """A device buffer of the library as a tensor (no copy)."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i8", "data": (ptr, False), "version": 2}


def _ntt1d_tables(logn):
    import ctypes
    pkg, n = _pkg(), 1 << logn
    q = np.zeros(1, np.uint64)
    pkg.call("cbs_get_primes", n, 54, 1, q.ctypes.data)
    host = [np.zeros(n, np.uint64) for _ in range(4)]
    ninv, mod = np.zeros(2, np.uint64), pkg.DModulus()
    pkg.call("cbs_ntt_tables_host", n, int(q[0]), *(h.ctypes.data for h in host), ninv.ctypes.data,
             ctypes.byref(mod))
    record = np.frombuffer(bytes(mod), np.uint64)
    rp, rps, irp, irps, ni, rec = (torch.from_numpy(h.view(np.int64).copy()).cuda() for h in (*host, ninv, record))
    return {"q": int(q[0]), "fwd": (rp, rps, rec), "inv": (irp, irps, rec, ni[0:1], ni[1:2])}


def _rns(case):
    pkg, n = _pkg(), 1 << case["logn"]
    size_q = case.get("size_q", case.get("limbs"))
    size_p = case.get("size_p", 1)

    def make():
        chain = np.zeros(size_q + size_p, np.uint64)
        pkg.call("cbs_get_primes", n, case["bits"], size_q + size_p, chain.ctypes.data)
        ctx = pkg.RnsContext(n, chain[:size_q], chain[size_q:])
        out = {"ctx": ctx, "chain": chain}
        if "level" in case:
            g = _gen(99)  # one switching key per digit, as the key owner uploads them
            out["evk"] = [_residues(g, (2,), chain, n) for _ in range(ctx.beta(size_q))]
            out["evk_ptrs"] = ctx.evk_array([e.data_ptr() for e in out["evk"]])
        return out

    got = _keep(("rns", n, case["bits"], size_q, size_p, "level" in case), make)
    if "level" in case:
        pkg.call("cbs_rns_prepare_level", got["ctx"].handle, case["level"])
    return got


def _gate_ctx(large, mode, mb):
    pkg = _pkg()

    def make():
        p = pkg.gate_default_params()
        if large:
            p.N, p.n = 2048, 630
        ctx = pkg.GateContext(p, max_batch=6144)
        ctx.keygen(7 + large)
        ctx.set_multibit(mb)
        ctx.set_fft_mode(mode)
        return ctx

    return _keep(("gate", large, mode, mb), make)


def _cbs_ctx(params, backend, mb, max_batch):
    pkg = _pkg()

    def make():
        ctx = pkg.Context(params=pkg.preset_params(params), max_batch=max_batch)
        ctx.set_br_backend({"ntt": pkg.BR_NTT, "split": pkg.BR_FFT64_SPLIT, "fft64": pkg.BR_FFT64}[backend])
        if mb > 1:
            ctx.set_br_multibit(mb)
        ctx.keygen_device(bytes(range(32)))
        return ctx

    return _keep(("cbs", params, backend, mb, max_batch), make)


_AES_KEY = bytes(range(16))


def _aes_ctx():
    pkg = _pkg()

    def make():
        ctx = _cbs_ctx("2x18", "fft64", 2, 128 * 16)
        pkg.call("cbs_aes128_setup_device", ctx.handle, _AES_KEY, bytes(range(64, 96)))
        return ctx

    return _keep("aes", make)


def _tcb_ctx(mb):
    pkg = _pkg()

    def make():
        ctx = pkg.TcbContext(max_batch=256)
        ctx.keygen(11)
        return ctx

    ctx = _keep("tcb", make)
    if _held.get("tcb_mb") != mb:
        ctx.set_multibit(mb)
        _held["tcb_mb"] = mb
    return ctx


def _tcb_z1():
    """The level-1 secret as the matrix of a -> a z1 mod X^N1 + 1 (float64, exact for 32-bit a)."""
    def make():
        ctx = _held["tcb"]
        z1 = torch.from_numpy(ctx.export_keys()["z1"].astype(np.float64)).cuda()
        n = len(z1)
        j, k = torch.arange(n, device="cuda").view(-1, 1), torch.arange(n, device="cuda").view(1, -1)
        return torch.where(k >= j, z1[(k - j) % n], -z1[(k - j) % n]).contiguous()

    return _keep("tcb_z1", make)


def prepare(case, seed):
    pkg, kind = _pkg(), case["kind"]
    rng = np.random.default_rng(int(seed))
    if kind == "ntt1d":
        n = 1 << case["logn"]
        t = _keep(("ntt1d", n), lambda: _ntt1d_tables(case["logn"]))
        x, z = (_residues(g, (case["polys"],), [t["q"]], n).view(case["polys"], n) for g in [_gen(seed)] * 2)
        return {"case": case, "t": t, "x": x, "z": z, "y": torch.empty_like(x), "w": torch.empty_like(z)}
    if kind == "ntt2d":
        r, g, n = _rns(case), _gen(seed), 1 << case["logn"]
        q = r["chain"][:case["limbs"]]
        return {"case": case, "r": r, "fwd": _residues(g, (case["polys"],), q, n),
                "inv": _residues(g, (case["polys"],), q, n)}
    if kind == "keyswitch":
        r, g, n = _rns(case), _gen(seed), 1 << case["logn"]
        q = r["chain"][:case["level"]]
        return {"case": case, "r": r, "c2": _residues(g, (case["count"],), q, n),
                "ct": _residues(g, (case["count"], 2), q, n)}
    if kind == "ckks":
        r, g, n = _rns(case), _gen(seed), 1 << case["logn"]
        q = r["chain"][:case["level"]]
        s = {"case": case, "r": r, "ct": _residues(g, (3,), q, n), "other": _residues(g, (2,), q, n)}
        s["scaled"] = torch.zeros((2, case["level"] - 1, n), dtype=torch.int64, device="cuda")
        return s
    if kind == "gate":
        ctx, count = _gate_ctx(0, case["mode"], case["mb"]), case["count"]
        ins = []
        for k in range(2):
            a, b = ctx.encrypt(rng.integers(0, 2, count).astype(np.uint8), seed=int(rng.integers(1 << 40)))
            ins += [_dev32(a), _dev32(b)]
        return {"case": case, "ctx": ctx, "in": ins,
                "out": (torch.zeros((count, ctx.params.n), dtype=torch.int32, device="cuda"),
                        torch.zeros(count, dtype=torch.int32, device="cuda"))}
    if kind == "ragged":
        s = {"case": case, "sets": []}
        for large, text in ((0, case["small"]), (1, case["large"])):
            ctx, reqs, keep, outs = _gate_ctx(large, case["mode"], case["mb"]), [], [], []
            for c in (int(v) for v in text.split(",")):
                a, b = ctx.encrypt(rng.integers(0, 2, c).astype(np.uint8), seed=int(rng.integers(1 << 40)))
                da, db = _dev32(a), _dev32(b)
                oa = torch.zeros((c, ctx.params.n), dtype=torch.int32, device="cuda")
                ob = torch.zeros(c, dtype=torch.int32, device="cuda")
                reqs.append((da.data_ptr(), db.data_ptr(), oa.data_ptr(), ob.data_ptr(), c))
                keep += [da, db]
                outs += [oa, ob]
            s["sets"].append((ctx, reqs, keep, outs))
        return s
    if kind == "aes":
        ctx, blocks = _aes_ctx(), case["blocks"]
        nonce = np.repeat(rng.integers(0, 256, (1, 12), dtype=np.uint8), blocks, axis=0)
        index = (int(rng.integers(1 << 24)) + np.arange(blocks, dtype=np.uint32)).astype(">u4")
        ctrs = np.ascontiguousarray(np.concatenate([nonce, index.view(np.uint8).reshape(blocks, 4)], axis=1))
        return {"case": case, "ctx": ctx, "ctrs": ctrs, "cipher": rng.integers(0, 256, (blocks, 16), dtype=np.uint8),
                "a": np.empty((blocks * 128, ctx.params.n), np.uint64), "b": np.empty(blocks * 128, np.uint64)}
    if kind == "cbs":
        ctx = _cbs_ctx(case["params"], case["backend"], case["mb"], 512)
        g, p = _gen(seed), ctx.params
        lwe = [torch.randint(0, int(p.q_lwe), shape, dtype=torch.int64, device="cuda", generator=g)
               for shape in ((case["count"], p.n), (case["count"],))]
        return {"case": case, "ctx": ctx, "a": lwe[0], "b": lwe[1]}
    ctx = _tcb_ctx(case["mb"])
    p = ctx.params
    a, b = ctx.encrypt(_tcb_bits(case, seed), seed=int(seed) + 3)
    return {"case": case, "ctx": ctx, "a": _dev32(a), "b": _dev32(b), "z1": _tcb_z1(),
            "rgsw": torch.zeros((case["count"], p.cb_levels, 2, 2, p.N1), dtype=torch.int32, device="cuda")}


def _tcb_bits(case, seed):
    return np.random.default_rng(int(seed)).integers(0, 2, case["count"]).astype(np.uint8)


# ---------------------------------------------------------------------------- one pass

def run(s):
    pkg, case = _pkg(), s["case"]
    kind = case["kind"]
    if kind == "ntt1d":
        n, t = 1 << case["logn"], s["t"]
        pkg.call("cbs_fnwt_1d_opt_outofplace_batched", s["y"].data_ptr(), s["x"].data_ptr(),
                 *(v.data_ptr() for v in t["fwd"]), n, case["polys"], None)
        pkg.call("cbs_inwt_1d_opt_outofplace_batched", s["w"].data_ptr(), s["z"].data_ptr(),
                 *(v.data_ptr() for v in t["inv"]), n, case["polys"], None)
        return s["y"], s["w"]
    if kind == "ntt2d":
        n, limbs = 1 << case["logn"], case["limbs"]
        for x, inverse in ((s["fwd"], 0), (s["inv"], 1)):
            pkg.call("cbs_rns_ntt_batched", s["r"]["ctx"].handle, x.data_ptr(), case["polys"], limbs * n, limbs, 0,
                     inverse, None)
        return s["fwd"], s["inv"]
    if kind == "keyswitch":
        pkg.call("cbs_rns_keyswitch_inplace", s["r"]["ctx"].handle, s["ct"].data_ptr(), s["c2"].data_ptr(),
                 s["r"]["evk_ptrs"], case["level"], case["count"], None)
        return s["ct"]
    if kind == "ckks":
        h, keys, level = s["r"]["ctx"].handle, s["r"]["evk_ptrs"], case["level"]
        if case["op"] == "rotate":
            pkg.call("cbs_ckks_rotate_inplace", h, s["ct"].data_ptr(), 5, keys, level, None)
            return s["ct"][:2]
        pkg.call("cbs_ckks_multiply_and_relin_inplace", h, s["ct"].data_ptr(), s["other"].data_ptr(), keys, level,
                 None)
        pkg.call("cbs_ckks_rescale_to_next", h, s["scaled"].data_ptr(), s["ct"].data_ptr(), 2, level, None)
        return s["ct"][:2], s["scaled"]
    if kind == "gate":
        oa, ob = s["out"]
        pkg.call("cbs_gate_eval_batch_device", s["ctx"].handle, pkg.GATE_NAND, *(t.data_ptr() for t in s["in"]),
                 case["count"], oa.data_ptr(), ob.data_ptr(), None)
        if case["mode"] == "fp64":  # every product rounds to the exact integer: the words are determined
            return oa, ob
        return s["ctx"].decrypt(oa.cpu().numpy().view(np.uint32), ob.cpu().numpy().view(np.uint32))
    if kind == "ragged":
        for ctx, reqs, _, _ in s["sets"]:  # a new request table per pass, as requests arrive
            ctx.ragged_plan(reqs)
            ctx.ragged_launch()
        return [t for _, _, _, outs in s["sets"] for t in outs]
    if kind == "aes":
        pkg.call("cbs_aes128_ctr_transcipher_ciphertext", s["ctx"].handle, s["ctrs"].ctypes.data,
                 s["cipher"].ctypes.data, case["blocks"], s["a"].ctypes.data, s["b"].ctypes.data)
        bits = np.empty(case["blocks"] * 128, np.uint8)
        pkg.call("cbs_lwe_decrypt_bits", s["ctx"].handle, s["a"].ctypes.data, s["b"].ctypes.data, len(bits),
                 s["a"].shape[1], bits.ctypes.data)
        return bits
    if kind == "cbs":
        import ctypes
        p, view = s["ctx"].params, ctypes.c_void_p()
        pkg.call("cbs_circuit_bootstrap_batch_device", s["ctx"].handle, s["a"].data_ptr(), s["b"].data_ptr(),
                 case["count"], p.n, ctypes.byref(view), None)
        return torch.as_tensor(_View(view.value, (case["count"], p.num_lut, 2, 2, p.N)), device="cuda")
    pkg.call("cbs_tcb_circuit_bootstrap_device", s["ctx"].handle, s["a"].data_ptr(), s["b"].data_ptr(), case["count"],
             None, s["rgsw"].data_ptr(), None)
    rows = s["rgsw"].view(-1, 2, s["rgsw"].shape[-1])  # the key owner's phases b - a z1, in [-1/2, 1/2)
    phase = (rows[:, 1].double() - rows[:, 0].double() @ s["z1"]) * 2.0 ** -32
    return (phase - torch.floor(phase + 0.5)).view(s["rgsw"].shape[:3] + s["rgsw"].shape[4:])


# ---------------------------------------------------------------------------- what a pass needs

def _ntt_flops(n, polys):
    """A multiply, an add and a subtract per butterfly."""
    return 1.5 * n * (n.bit_length() - 1) * polys


def _keyswitch_work(n, level, size_p, count):
    beta, qlp = -(-level // size_p), level + size_p
    transforms = level + beta * qlp - level + 2 * size_p + 2 * level
    flops = count * (_ntt_flops(n, transforms) + 2.0 * n * (beta * qlp * size_p + 2 * beta * qlp + 2 * level * size_p))
    return {"bytes": 8.0 * n * (2 * beta * qlp + count * (level + 4 * level)), "flops": flops}


def _rotation_work(n, steps, N, digits, cols=2):
    """Blind rotation: per coefficient 2*digits forward and 2 inverse N/2-point complex transforms
    and 2*digits*cols spectrum products."""
    m = N // 2
    return n * steps * ((2 * digits + cols) * 5.0 * m * math.log2(m) + 2 * digits * cols * 8.0 * m)


def work(case):
    kind, n = case["kind"], 1 << case.get("logn", 0)
    if kind == "ntt1d":
        return {"bytes": 8.0 * n * (4 * case["polys"] + 4), "flops": _ntt_flops(n, 2 * case["polys"])}
    if kind == "ntt2d":
        polys = case["polys"] * case["limbs"]
        return {"bytes": 8.0 * n * (4 * polys + 2 * case["limbs"]), "flops": _ntt_flops(n, 2 * polys)}
    if kind == "keyswitch":
        return _keyswitch_work(n, case["level"], case["size_p"], case["count"])
    if kind == "ckks":
        w = _keyswitch_work(n, case["level"], case["size_p"], 1)
        if case["op"] == "mul":
            w["bytes"] += 8.0 * n * (2 * case["level"] + 2 * (case["level"] - 1))
            w["flops"] += _ntt_flops(n, 2 * case["level"]) + 10.0 * n * case["level"]
        return w
    if kind in ("gate", "ragged"):
        sets = [(1024, 636, case["count"], 2)] if kind == "gate" else [
            (N, n, sum(int(v) for v in case[k].split(",")), 1) for N, n, k in ((1024, 636, "small"), (2048, 630, "large"))]
        b = f = 0.0
        for N, n, count, inputs in sets:
            ksk = 4.0 * N * 8 * 3 * (n + 1)
            b += 16.0 * n * 6 * 2 * (N // 2) + ksk + 4.0 * count * (n + 1) * (inputs + 1)
            f += _rotation_work(n, count, N, 3) + 2.0 * count * N * 8 * (n + 1)
        return {"bytes": b, "flops": f}
    if kind == "aes":
        bits = 1280.0 * case["blocks"]  # ten rounds of 128 bootstraps
        keys = 16.0 * 630 * 4 * 2 * 1024 + 2.0 * 2 * 2048 * 127 * 631 + 8.0 * 8 * 256 * 2 * 2048
        trace = bits * 4 * (12 * (5 + 3) * 51200.0 + 12 * 15 * 8192.0)
        cmux = 160.0 * case["blocks"] * 255 * (10 * 51200.0 + 16 * 8192.0)
        return {"bytes": keys + 8.0 * 128 * case["blocks"] * 631,
                "flops": _rotation_work(630, bits, 2048, 2) + trace + cmux + bits * 2 * 2048 * 2 * 631}
    if kind == "cbs":
        digits = 3 if case["params"] == "3x12" else 2
        c = case["count"]
        return {"bytes": 8.0 * 630 * 2 * digits * 2 * 2048 + 8.0 * c * (631 + 16 * 2048),
                "flops": _rotation_work(630, c, 2048, digits) + c * 4 * _ntt_flops(2048, 12 * 6)}
    c = case["count"]
    return {"bytes": 16.0 * 630 * 6 * 2 * 1024 + 4.0 * 2 * 2049 * 8 * 15 * 2048 + 4.0 * c * (631 + 3 * 4 * 1024),
            "flops": _rotation_work(630, 3.0 * c, 2048, 3) + 6.0 * c * 2049 * 8 * 2048}


def tolerance(case):
    # tcb: the row phases carry the bootstrapping noise (2^-18 of the torus, beside messages up to
    # 2^-6); another rounding of the FP64 products gives another sample of it
    return {"rel": 8e-3, "max": 0.08} if case["kind"] == "tcb" else "exact"


def exact(case, seed):
    if case["kind"] != "tcb":
        return None  # whole numbers, compared word for word
    prepare(case, seed)
    p, z1 = _held["tcb"].params, _held["tcb"].export_keys()["z1"].astype(np.float64)
    bits = _tcb_bits(case, seed)
    out = np.zeros((case["count"], p.cb_levels, 2, p.N1))
    for k in range(p.cb_levels):
        g = 2.0 ** (-(k + 1) * p.cb_bits)
        out[:, k, 0, :] = -g * bits[:, None] * z1[None]  # row 2k: -m g_k z1
        out[:, k, 1, 0] = g * bits  # row 2k + 1: m g_k
    return out
