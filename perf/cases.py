"""Performance cases of the CKKS engine: the calls a program that computes on
encrypted data makes, through the public entry points of the package.

Everything is seeded. Ciphertexts, evaluation keys and encoded plaintexts are
uniform residues below each limb's prime, which is what they look like in the
evaluation domain; evaluation keys, plaintext tables, packed weights and output
buffers are held by the program across calls, so prepare() makes them.
All results are residues (32-bit words) and have to be the same words.
"""
import functools
import importlib
import json
import math
import os

import numpy as np
import torch

N = 1 << 16            # ring degree of every parameter set
LIMB = 4 * N           # bytes of one limb
MAX_LEVEL = {"bootparam_40": 28, "bootparam_35": 31, "bootparam_30": 34}


def listed():
    return [
        # Sum of two nearly exhausted ciphertexts: the smallest call, all latency.
        {"name": "add_level1", "kind": "add", "params": "bootparam_40", "level": 1},
        # Masking or weighting by a plaintext, then rescaling, half way down the
        # levels that remain after bootstrapping (13).
        {"name": "pmult_rescale_level7", "kind": "pmult", "params": "bootparam_40", "level": 7},
        # Batched transform, forward and inverse: 16 polynomials of 40 limbs (the
        # benchmark's first workload, the largest transform).
        {"name": "ntt_16x40", "kind": "ntt", "polys": 16, "limbs": 40},
        # One polynomial of an ordinary ciphertext there and back (23 limbs: level 16,
        # the default encryption level of bootparam_40).
        {"name": "ntt_1x23", "kind": "ntt", "polys": 1, "limbs": 23},
        # Product of two fresh ciphertexts at the top level with relinearisation and
        # rescale (the benchmark's headline).
        {"name": "hmult_level28", "kind": "hmult", "params": "bootparam_40", "level": 28, "rescale": True},
        # The same near the end of a computation, 9 limbs: launches and latency count.
        {"name": "hmult_level5", "kind": "hmult", "params": "bootparam_40", "level": 5, "rescale": True},
        # One rotation (key switch, then the automorphism) at the default encryption
        # level of another parameter set.
        {"name": "rotate_level19_35", "kind": "rotate", "params": "bootparam_35", "level": 19},
        # 64 rotations of one ciphertext sharing a decomposition (convolutions, matrix
        # products; the benchmark's rotation sweep).
        {"name": "hoisted64_level28", "kind": "hoisted", "params": "bootparam_40", "level": 28, "rotations": 64},
        # One CoeffToSlot group of bootstrapping: 31 diagonals as 16 baby and 2 giant steps.
        {"name": "transform_16x2_level27", "kind": "transform", "params": "bootparam_40", "level": 27,
         "baby": 16, "giant": 2},
        # The double-angle steps that end bootstrapping's modular reduction
        # (x <- 2 x^2 - 1, three levels): a chain of dependent small operators.
        {"name": "double_angle_level16", "kind": "double_angle", "params": "bootparam_40", "level": 16, "steps": 3},
        # Query projection of an encrypted BERT-base layer: 768 features to 768.
        {"name": "project_768x768_level11", "kind": "project", "params": "bootparam_40", "level": 11,
         "n_in": 768, "n_out": 768},
        # Encoding and encrypting one message at the default encryption level, from
        # host coefficients.
        {"name": "encrypt_level16", "kind": "encrypt", "params": "bootparam_40", "level": 16},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["add", "pmult", "ntt", "ntt", "hmult", "hmult", "rotate", "hoisted", "transform",
                       "double_angle", "project", "encrypt"])
    if kind == "ntt":
        return {"kind": kind, "polys": _log_int(rng, 1, 16), "limbs": _log_int(rng, 1, 40)}
    params = rng.choice(["bootparam_40", "bootparam_40", "bootparam_35", "bootparam_30"])
    top = MAX_LEVEL[params]
    case = {"kind": kind, "params": params}
    if kind == "hmult":
        case.update(level=rng.randint(1, top), rescale=rng.random() < 0.75)
    elif kind == "hoisted":
        case.update(level=rng.randint(2, min(top, 28)), rotations=_log_int(rng, 2, 40))
    elif kind == "transform":
        case.update(level=rng.randint(4, top), baby=rng.randint(2, 16), giant=rng.randint(1, 4))
    elif kind == "double_angle":
        steps = rng.randint(1, 4)
        case.update(level=rng.randint(steps, top), steps=steps)
    elif kind == "project":
        case.update(level=rng.randint(2, 11), n_in=_log_int(rng, 16, 768), n_out=_log_int(rng, 16, 768))
    else:
        case.update(level=rng.randint(1, top))
    return case


@functools.lru_cache(maxsize=None)
def _engine(params):
    """One context per parameter set for the life of the program."""
    pkg = importlib.import_module("cheddar-fhe_b200")
    p = pkg.load_params(params + ".json")
    return pkg.Engine(p), p


class _Residues:
    """Uniform residues of a limb list, from one seed."""

    def __init__(self, eng, seed):
        self.eng = eng
        self.gen = torch.Generator(device=f"cuda:{eng.device}").manual_seed(seed)

    def __call__(self, gidx, *lead):
        out = self.eng.empty(*lead, len(gidx), N)
        for i, g in enumerate(gidx):
            out[..., i, :] = torch.randint(0, int(self.eng.primes[g]), (*lead, N), dtype=torch.int32,
                                           device=out.device, generator=self.gen)
        return out


def _key_limbs(p):
    return list(range(len(p["terminal_primes"]) + len(p["main_primes"]) + len(p["auxiliary_primes"])))


def _distances(rng, count):
    """Rotation distances: powers of two first, then random ones."""
    rots = [1 << i for i in range(min(15, count))]
    while len(rots) < count:
        r = int(rng.integers(1, N // 2))
        if r not in rots:
            rots.append(r)
    return rots


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    s.eng, p = eng, p = _engine(case.get("params", "bootparam_40"))
    rng = np.random.default_rng(seed)
    rand = _Residues(eng, seed)
    s.main = len(p["main_primes"])
    if s.kind == "ntt":
        s.g = list(range(case["limbs"]))
        s.src = rand(s.g, case["polys"])
        s.mid, s.out = torch.empty_like(s.src), torch.empty_like(s.src)
        return s
    s.level = level = case["level"]
    s.g = eng.level_limbs(level)
    nq = len(s.g)
    max_beta = eng.beta(MAX_LEVEL[case["params"]])
    if s.kind == "add":
        s.x, s.y = rand(s.g, 2), rand(s.g, 2)
        s.out = torch.empty_like(s.x)
    elif s.kind == "pmult":
        s.x, s.pt = rand(s.g, 2), rand(s.g)
        s.prod = torch.empty_like(s.x)
        s.out = eng.empty(2, len(eng.level_limbs(level - 1)), N)
    elif s.kind == "hmult":
        s.rescale = case["rescale"]
        s.x, s.y = rand(s.g, 2), rand(s.g, 2)
        s.key = rand(_key_limbs(p), 2, max_beta)
        s.out = eng.empty(2, len(eng.level_limbs(level - 1)) if s.rescale else nq, N)
    elif s.kind == "rotate":
        s.rot = int(rng.integers(1, N // 2))
        s.x = rand(s.g, 2)
        s.key = rand(_key_limbs(p), 2, max_beta)
        s.switched = eng.empty(2, nq, N)
        s.out = eng.empty(2, nq, N)
    elif s.kind == "hoisted":
        s.rots = _distances(rng, case["rotations"])
        s.x = rand(s.g, 2)
        key = rand(_key_limbs(p), len(s.rots), 2, eng.beta(level))
        s.kb = [list(k[0]) for k in key]
        s.ka = [list(k[1]) for k in key]
        s.out = eng.empty(len(s.rots), 2, nq, N)
    elif s.kind == "transform":
        nb, ng = case["baby"], case["giant"]
        stride = 1 << int(rng.integers(0, 9))
        s.baby = [i * stride for i in range(nb)]
        s.giant = [j * nb * stride for j in range(ng)]
        key = rand(_key_limbs(p), nb + ng, 2, max_beta)
        s.baby_keys = [None if r == 0 else (list(key[i][0]), list(key[i][1])) for i, r in enumerate(s.baby)]
        s.giant_keys = [None if r == 0 else (list(key[nb + j][0]), list(key[nb + j][1]))
                        for j, r in enumerate(s.giant)]
        pts = rand(eng.level_limbs(level, eng.alpha), ng, nb)
        # an odd number of diagonals leaves the last place of the last giant step empty
        s.pts = [[pts[j][i] if ng == 1 or (j, i) != (ng - 1, nb - 1) else None for i in range(nb)] for j in range(ng)]
        s.x = rand(s.g, 2)
        s.out = eng.empty(2, len(eng.level_limbs(level - 1)), N)
    elif s.kind == "double_angle":
        s.x = rand(s.g, 2)
        s.key = rand(_key_limbs(p), 2, max_beta)
        s.steps = []
        for k in range(case["steps"]):
            g = eng.level_limbs(level - k - 1)
            one = np.array([rng.integers(0, int(eng.primes[gi])) for gi in g], dtype=np.uint32)
            s.steps.append((level - k, g, one, eng.empty(2, len(g), N), eng.empty(2, len(g), N)))
    elif s.kind == "project":
        n_in, n_out = case["n_in"], case["n_out"]
        s.x = rand(s.g, n_in)
        s.out = eng.empty(n_out, nq, N)
        s.xs, s.ys = list(s.x), list(s.out)
        w = np.stack([rng.integers(0, int(eng.primes[gi]), (n_in, n_out), dtype=np.uint32) for gi in s.g])
        s.packed = eng.gemm_pack_weights(w, s.g)
    elif s.kind == "encrypt":
        # slots of order one at scale 2^40 spread over 2^16 coefficients; a normal error of 3.2
        s.coeffs = rng.normal(0.0, 2.0 ** 32, N)
        s.seed, s.sigma = int(seed), 3.2
        s.secret = rand(s.g)
        s.m, s.e, s.e_ntt, s.b, s.a = (eng.empty(nq, N) for _ in range(5))
    else:
        raise ValueError(s.kind)
    return s


def run(s):
    eng = s.eng
    if s.kind == "ntt":
        eng.ntt_(s.mid, s.src, s.g)
        eng.intt_(s.out, s.mid, s.g, mont_keep=True)
        return s.mid, s.out
    if s.kind == "add":
        eng.elementwise_multi_(False, 0, [s.out[0], s.out[1]], [s.x[0], s.x[1]], [s.y[0], s.y[1]], None, s.g)
        return s.out
    if s.kind == "pmult":
        eng.elementwise_multi_(False, 3, [s.prod[0], s.prod[1]], [s.x[0], s.x[1]], [s.pt, s.pt], None, s.g)
        eng.moddown_(s.level, 1, s.out, s.prod)
        return s.out
    if s.kind == "hmult":
        eng.hmult_(s.level, s.out[0], s.out[1], s.x[0], s.x[1], s.y[0], s.y[1], list(s.key[0]), list(s.key[1]),
                   s.main, s.rescale)
        return s.out
    if s.kind == "rotate":
        eng.keyswitch_(s.level, s.switched[0], s.switched[1], s.x[1], s.x[0], list(s.key[0]), list(s.key[1]), s.main)
        galois = eng.galois(s.rot)
        eng.permute_(s.out[0], s.switched[0], None, galois, s.g)
        eng.permute_(s.out[1], s.switched[1], None, galois, s.g)
        return s.out
    if s.kind == "hoisted":
        eng.hoisted_rotations_(s.level, s.out, s.x[0], s.x[1], s.rots, s.kb, s.ka, s.main)
        return s.out
    if s.kind == "transform":
        eng.linear_transform_(s.level, s.out[0], s.out[1], s.x[0], s.x[1], s.baby, s.baby_keys, s.giant,
                              s.giant_keys, s.pts, s.main)
        return s.out
    if s.kind == "double_angle":
        kb, ka = list(s.key[0]), list(s.key[1])
        x = s.x
        for level, g, one, square, out in s.steps:
            eng.hmult_(level, square[0], square[1], x[0], x[1], x[0], x[1], kb, ka, s.main)
            eng.elementwise_multi_(False, 0, [out[0], out[1]], [square[0], square[1]], [square[0], square[1]],
                                   None, g)
            eng.const_op_(1, out[0], out[0], None, one, g)
            x = out
        return x
    if s.kind == "project":
        eng.ctpt_gemm_(s.ys, s.xs, s.packed, s.g)
        return s.out
    if s.kind == "encrypt":
        eng.encode_coeffs_(s.m, s.coeffs, s.g)
        eng.sample_uniform_(s.a, s.g, s.seed, 1)
        eng.sample_error_(s.e, s.g, s.sigma, s.seed, 2)
        eng.ntt_(s.e_ntt, s.e, s.g, mont_conv=True)
        eng.encrypt_(s.b, s.a, s.secret, s.e_ntt, s.m, s.g)
        return s.m, s.b, s.a
    raise ValueError(s.kind)


def work(case):
    """Compulsory traffic: operands, keys, tables and results once each; for the
    projection also the 8-bit multiply-adds (two operations each) that an exact
    product of 32-bit words by byte planes takes."""
    kind = case["kind"]
    if kind == "ntt":
        return {"bytes": 4 * case["polys"] * case["limbs"] * LIMB, "flops": 0}
    with open(os.path.join("cheddar-fhe_b200", "parameters", case["params"] + ".json")) as f:
        p = json.load(f)
    alpha, ter = len(p["auxiliary_primes"]), len(p.get("terminal_primes") or [])
    level = case["level"]

    def limbs(lv):
        return sum(p["level_config"][lv])

    def digits(lv):
        return -(-(p["level_config"][lv][0] + ter) // alpha)

    nq = limbs(level)
    key = 2 * digits(level) * (nq + alpha)
    flops = 0
    if kind == "add":
        n = 6 * nq
    elif kind == "pmult":
        n = 3 * nq + 2 * limbs(level - 1)
    elif kind == "hmult":
        n = 4 * nq + key + 2 * limbs(level - 1 if case["rescale"] else level)
    elif kind == "rotate":
        n = 4 * nq + key
    elif kind == "hoisted":
        n = 2 * nq + case["rotations"] * (key + 2 * nq)
    elif kind == "transform":
        nb, ng = case["baby"], case["giant"]
        n = 2 * nq + (nb + ng - 2) * key + (nb * ng - (ng > 1)) * (nq + alpha) + 2 * limbs(level - 1)
    elif kind == "double_angle":
        n = 2 * nq + 2 * limbs(level - case["steps"])
        n += max(2 * digits(lv) * (limbs(lv) + alpha) for lv in range(level - case["steps"] + 1, level + 1))
    elif kind == "project":
        n_in, n_out = case["n_in"], case["n_out"]
        n = (n_in + n_out) * nq
        flops = 2 * 16 * n_in * n_out * N * nq
    else:  # encrypt: the coefficients and the secret in, message and both parts out
        n = 4 * nq + 2
    return {"bytes": n * LIMB, "flops": flops}


def tolerance(case):
    return "exact"
