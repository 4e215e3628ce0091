"""The work that a program built on this library has it do, case by case, through its public calls.

listed() holds one case for each use, draw() more of the same ranges. Kinds of case:

  msm     an MSM on device buffers: a commitment to a polynomial whose coefficients are on the GPU.
          form "device" passes the bases with each call, "resident" keeps an uploaded base set,
          "host" is the drop-in call of a program whose arrays lie in ordinary host memory.
  ntt     one forward or inverse transform between device buffers
  fr      one element-wise operation or batch inversion over a vector of Fr on the device
  g1_fft  a group FFT (Lagrange basis of a structured reference string)
  binary  sums of selected bases for many 0/1 rows (commitments to witness bits)
  batch   many MSMs against one base set and many NTTs, planned once and run again and again

Sizes follow the tests and the benchmark of this repository: MSMs of 2^10 to 2^22 points, NTTs of
2^10 to 2^24 elements, both curves, sizes that are no power of two wherever the call allows them.
All results are integers; they have to be the same to the bit, so exact() gives no values.
"""
import ctypes
import importlib
import random

import numpy as np
import torch

zk = importlib.import_module("zikkurat-algebra_b200")

BN, BLS = zk.BN254, zk.BLS12_381
KINDS = {"affine": zk.OUT_AFFINE, "proj": zk.OUT_PROJ, "jac": zk.OUT_JAC}


def listed():
    return [
        # the smallest commitments: launches, synchronisation and the host's share count
        {"name": "msm_bn_1000", "kind": "msm", "curve": BN, "form": "device", "n": 1000, "mont": False, "out": "affine"},
        # a mid-sized circuit's commitment against an uploaded setup
        {"name": "msm_bn_2p16_resident", "kind": "msm", "curve": BN, "form": "resident", "n": 65536, "mont": True, "out": "affine"},
        # the drop-in call on ordinary (pageable) host arrays, bases copied each time, odd size
        {"name": "msm_bn_300k_host", "kind": "msm", "curve": BN, "form": "host", "n": 300007, "mont": True, "out": "proj"},
        # a large commitment over the wider curve, odd size
        {"name": "msm_bls_1m", "kind": "msm", "curve": BLS, "form": "device", "n": 1000003, "mont": True, "out": "jac"},
        # the benchmark's MSM
        {"name": "msm_bn_2p22", "kind": "msm", "curve": BN, "form": "device", "n": 1 << 22, "mont": True, "out": "affine"},
        # a small transform, where one or two launches are all there is
        {"name": "ntt_bls_2p12_fwd", "kind": "ntt", "curve": BLS, "m": 12, "inverse": False},
        # evaluations back to coefficients at a mid-sized circuit
        {"name": "ntt_bn_2p18_inv", "kind": "ntt", "curve": BN, "m": 18, "inverse": True},
        # the benchmark's NTT
        {"name": "ntt_bn_2p24_fwd", "kind": "ntt", "curve": BN, "m": 24, "inverse": False},
        # denominators of a lookup or permutation argument
        {"name": "fr_inv_bls_1m", "kind": "fr", "curve": BLS, "op": "inv", "n": 1000001},
        # Lagrange-basis setup
        {"name": "g1_fft_bn_2p14_inv", "kind": "g1_fft", "curve": BN, "m": 14, "inverse": True, "jac": False},
        # witness-bit columns
        {"name": "binary_bn_64x2p18", "kind": "binary", "curve": BN, "rows": 64, "n": 1 << 18, "out": "affine"},
        # a prover's round: mixed MSMs and NTTs as one planned batch
        {"name": "batch_bn_12_12", "kind": "batch", "curve": BN, "msms": 12, "ntts": 12, "log_max": 18, "mix": 1},
    ]


def _log_uniform(rng, lo, hi):
    return int(2 ** rng.uniform(lo, hi))


def draw(rng):
    kind = rng.choice(["msm", "msm", "msm", "ntt", "ntt", "fr", "g1_fft", "binary", "batch"])
    curve = rng.choice([BN, BLS])
    if kind == "msm":
        form = rng.choice(["device", "resident", "host"])
        top = 19 if form == "host" else 22 if curve == BN else 20
        return {"kind": kind, "curve": curve, "form": form, "n": _log_uniform(rng, 10, top),
                "mont": rng.random() < 0.7, "out": rng.choice(["affine", "proj", "jac"])}
    if kind == "ntt":
        return {"kind": kind, "curve": curve, "m": rng.randint(10, 24), "inverse": rng.random() < 0.5}
    if kind == "fr":
        return {"kind": kind, "curve": curve, "op": rng.choice(["inv", "mul"]), "n": _log_uniform(rng, 14, 22)}
    if kind == "g1_fft":
        return {"kind": kind, "curve": curve, "m": rng.randint(9, 14 if curve == BN else 11),
                "inverse": rng.random() < 0.5, "jac": rng.random() < 0.5}
    if kind == "binary":
        return {"kind": kind, "curve": curve, "rows": rng.randint(1, 64), "n": _log_uniform(rng, 12, 18),
                "out": rng.choice(["affine", "proj", "jac"])}
    return {"kind": kind, "curve": curve, "msms": rng.randint(2, 16), "ntts": rng.randint(2, 16),
            "log_max": rng.randint(14, 18), "mix": rng.randint(2, 1 << 20)}


# ----------------------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _fr(curve, n, g):
    """(n, 4) limbs of field elements, uniform below the largest multiple of 2^192 under the order"""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    x[:, 3] = torch.randint(0, zk.R_MOD[curve] >> 192, (n,), dtype=torch.int64, device="cuda", generator=g)
    return x


def _bases(curve, n, g):
    """n affine points k G with random k"""
    out = torch.empty((n, 2 * zk.NLIMBS_P[curve]), dtype=torch.int64, device="cuda")
    ks = _fr(curve, n, g)
    torch.cuda.synchronize()
    zk.g1_gen_mul_device(curve, n, ks, out)
    torch.cuda.synchronize()
    return out


def _host(t):
    return t.cpu().numpy().view(np.uint64)


def _batch_sizes(case):
    r = random.Random(case["mix"])
    msms = [_log_uniform(r, 10, case["log_max"]) for _ in range(case["msms"])]
    ntts = [(r.randint(12, case["log_max"] + 2), r.random() < 0.5) for _ in range(case["ntts"])]
    return msms, ntts


def prepare(case, seed):
    g, curve, kind = _generator(seed), case["curve"], case["kind"]
    nlp = zk.NLIMBS_P[curve]
    s = {"case": case}
    if kind == "msm":
        s["scalars"], s["bases"] = _fr(curve, case["n"], g), _bases(curve, case["n"], g)
        if case["form"] == "host":
            s["scalars"], s["bases"] = _host(s["scalars"]), _host(s["bases"])
        elif case["form"] == "resident":
            s["set"] = zk.Bases(curve, s["bases"])
    elif kind == "ntt":
        s["gen"] = zk.fft_subgroup(curve, case["m"])
        s["x"] = _fr(curve, 1 << case["m"], g)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "fr":
        s["a"], s["b"] = _fr(curve, case["n"], g), _fr(curve, case["n"], g)
        s["y"] = torch.empty_like(s["a"])
    elif kind == "g1_fft":
        n = 1 << case["m"]
        one = np.array(zk.to_limbs((1 << (64 * nlp)) % zk.P_MOD[curve], nlp)).view(np.int64)
        z = torch.from_numpy(one).cuda().expand(n, nlp)
        s["gen"] = zk.fft_subgroup(curve, case["m"])
        s["x"] = torch.cat([_bases(curve, n, g), z], dim=1).contiguous()
        s["y"] = torch.empty_like(s["x"])
    elif kind == "binary":
        s["bits"] = torch.randint(0, 2, (case["rows"], case["n"]), dtype=torch.uint8, device="cuda", generator=g)
        s["bases"] = _bases(curve, case["n"], g)
        s["y"] = torch.empty((case["rows"], (2 if case["out"] == "affine" else 3) * nlp), dtype=torch.int64, device="cuda")
    else:
        msms, ntts = _batch_sizes(case)
        s["set"] = zk.Bases(curve, _bases(curve, max(msms), g))
        b = zk.Batch(curve, s["set"])
        s["points"] = [b.add_msm(n, _fr(curve, n, g)) for n in msms]
        s["values"] = []
        for m, inverse in ntts:
            x = _fr(curve, 1 << m, g)
            s["values"].append(torch.empty_like(x))
            b.add_ntt(m, x, s["values"][-1], inverse=inverse)
        s["batch"] = b
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    curve, kind = case["curve"], case["kind"]
    if kind == "msm":
        out = KINDS[case["out"]]
        if case["form"] == "device":
            return zk.msm_device(curve, case["n"], s["scalars"], s["bases"], mont=case["mont"], kind=out)
        if case["form"] == "resident":
            return s["set"].msm(case["n"], s["scalars"], mont=case["mont"], kind=out)
        call = {"affine": zk.msm_affine, "jac": zk.msm_jac}.get(case["out"])
        if call:
            return call(curve, s["scalars"], s["bases"], mont=case["mont"])
        return (zk.msm if case["mont"] else zk.msm_std)(curve, s["scalars"], s["bases"])
    if kind == "ntt":
        zk.ntt_device(curve, case["m"], s["x"], s["y"], inverse=case["inverse"], gen=s["gen"])
        return s["y"]
    if kind == "fr":
        p = [ctypes.c_void_p(s["a"].data_ptr()), ctypes.c_void_p(s["b"].data_ptr() if case["op"] == "mul" else None)]
        status = zk.lib().zkg_fr_map_device(curve, zk.FR_OPS[case["op"]], case["n"], *p, None, None, None,
                                            ctypes.c_void_p(s["y"].data_ptr()))
        if status:
            raise zk.ZkgError("zkg_fr_map_device", status)
        return s["y"]
    if kind == "g1_fft":
        zk.g1_fft_device(curve, case["m"], s["x"], s["y"], inverse=case["inverse"], gen=s["gen"], jac=case["jac"])
        return s["y"]
    if kind == "binary":
        zk.msm_binary_device(curve, case["rows"], case["n"], s["bits"], case["n"], s["bases"], s["y"], kind=KINDS[case["out"]])
        return s["y"]
    s["batch"].run()
    return s["points"] + s["values"]


def exact(case, seed):
    """No floating outputs: every result is an integer, the same to the bit whoever computes it."""
    return None


# ------------------------------------------------------------------------------------- work

def _product(words):
    """multiplications and additions of machine words in one Montgomery product"""
    return 2 * (2 * words * words + words)


def _msm(curve, n):
    """Pippenger with windows of about log2(n) bits: a mixed addition (10 products) a window and point"""
    windows = -(-254 // max(n.bit_length() - 1, 1))
    return {"bytes": n * (32 + 16 * zk.NLIMBS_P[curve]), "flops": n * windows * 10 * _product(zk.NLIMBS_P[curve])}


def _ntt(m):
    return {"bytes": 64 << m, "flops": (m << m) // 2 * _product(4)}


def work(case):
    kind, nlp = case["kind"], zk.NLIMBS_P[case["curve"]]
    if kind == "msm":
        return _msm(case["curve"], case["n"])
    if kind == "ntt":
        return _ntt(case["m"])
    if kind == "fr":
        inv = case["op"] == "inv"
        return {"bytes": case["n"] * (64 if inv else 96), "flops": case["n"] * (3 if inv else 1) * _product(4)}
    if kind == "g1_fft":
        # a butterfly multiplies a point by a 254-bit scalar: about 250 doublings and additions in all
        n = 1 << case["m"]
        return {"bytes": n * 48 * nlp, "flops": (n // 2) * case["m"] * 250 * 8 * _product(nlp)}
    if kind == "binary":
        # subset sums of eight columns, one addition a row and eight columns
        return {"bytes": case["n"] * (case["rows"] + 16 * nlp), "flops": case["n"] * (32 + case["rows"] / 8) * 10 * _product(nlp)}
    msms, ntts = _batch_sizes(case)
    parts = [_msm(case["curve"], n) for n in msms] + [_ntt(m) for m, _ in ntts]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
