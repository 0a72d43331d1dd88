"""The work a user of this framework has it do, as measured cases.

The search for the smallest irreducible factor of x^r + x^s + 1 over GF(2)
has four kinds of device work, each called through the public entry points of
`mersenne_trinomial_b200`: the Zech-log sieve over all s, repeated squaring of
many residues, products of long polynomials (by themselves, in batches, and as
the running product of the per-degree scan), and gcds; `scan` is the whole
deep search over sieve survivors.  Sizes are those of the package's own
workloads, tests and benchmark (r = 44687, r ~ 10^5, r ~ 10^6,
r = 136279841), with odd and ragged ones between them.

A case is a dict with a "kind" and that kind's sizes:

  sieve      r, dmin, dmax, smax       best[] over s = 0..smax (device)
  square     r, states, k              k squarings of each resident state
  frobenius  r, states, k              the same from x, host s in, host F_k out
  stage2     r, degrees                square and running product, one s
  mul        abits, bbits              one product on device buffers
  mulbatch   jobs, lo, hi, sizes       products of 2^lo .. 2^hi bit operands,
                                       lengths drawn by `sizes`
  fft        m                         one forward and one inverse transform
  gcd        bits, pairs, common       half-gcd gcds in one lockstep batch
  scan       r, ns, k0, maxd, L0, block   deep scan, result lines

Every result is a bit string or a whole number, so outputs are compared for
equality and `exact` has no 64-bit value to offer for any of them.
"""
from __future__ import annotations

import numpy as np
import torch

import mersenne_trinomial_b200 as M
from mersenne_trinomial_b200 import engine as E
from mersenne_trinomial_b200 import workloads as W

R_DEEP = W.R_DEEP
DEV = "cuda"


def listed():
    return [
        # the stage-1 sieve of a small exponent: all s, degrees 2..20
        {"name": "sieve_small", "kind": "sieve", "r": 44687, "dmin": 2, "dmax": 20, "smax": 22343},
        # stage 1 at the record exponent: every s <= r/2, degrees 2..24
        {"name": "sieve_full", "kind": "sieve", "r": R_DEEP, "dmin": 2, "dmax": 24,
         "smax": R_DEEP // 2},
        # per-degree squaring of many small residues, which stay in L2
        {"name": "square_mid", "kind": "square", "r": 999961, "states": 256, "k": 64},
        # the headline: 64 residues at the record exponent
        {"name": "square_deep", "kind": "square", "r": R_DEEP, "states": 64, "k": 16},
        # the host-buffer call: s values in, F_k out, for a ragged few
        {"name": "frobenius_host", "kind": "frobenius", "r": R_DEEP, "states": 7, "k": 65},
        # the smallest calls: one s, a few words, launches and latency
        {"name": "stage2_small", "kind": "stage2", "r": 44687, "degrees": 8},
        # one s at the record exponent, a degree at a time
        {"name": "stage2_deep", "kind": "stage2", "r": R_DEEP, "degrees": 2},
        # one short uneven product
        {"name": "mul_ragged", "kind": "mul", "abits": 70001, "bbits": 51203},
        # 64 uneven products, 2^16 .. 2^27 bits an operand
        {"name": "mul_batch", "kind": "mulbatch", "jobs": 64, "lo": 16.0, "hi": 27.0,
         "sizes": 1},
        # the transforms by themselves (both directions), an ordinary size
        {"name": "fft_m20", "kind": "fft", "m": 20},
        # interval gcds of resident survivors at r ~ 10^6
        {"name": "gcd_batch", "kind": "gcd", "bits": 1000183, "pairs": 8, "common": 131},
        # a whole deep scan of a small exponent, interval gcds included
        {"name": "scan_small", "kind": "scan", "r": 99767, "ns": 24, "k0": 16, "maxd": 144,
         "L0": 64, "block": 1},
    ]


def _logint(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(float(lo) * (float(hi) / lo) ** rng.random()))))


def _sieve_prime(start, dmax):
    """The next r the sieve accepts (prime, +-1 mod 8, coprime to every 2^d - 1)."""
    r = start | 1
    while not (r % 8 in (1, 7) and W.is_prime(r) and W.sieve_compatible(r, dmax)):
        r += 2
    return r


def draw(rng):
    kind = rng.choice(["sieve", "square", "square", "frobenius", "stage2", "mul", "mul",
                       "mulbatch", "fft", "gcd", "scan"])
    if kind == "sieve":
        dmax = rng.randint(14, 24)
        r = _sieve_prime(_logint(rng, 40000, 130_000_000), dmax)
        smax = _logint(rng, r // 20, r // 2)
        return {"kind": kind, "r": r, "dmin": rng.choice([2, 2, rng.randint(2, dmax)]),
                "dmax": dmax, "smax": smax}
    if kind == "square":
        r = _logint(rng, 4001, R_DEEP) | 1
        nw = (r + 63) // 64
        states = _logint(rng, 1, max(1, min(256, 64 * 2129373 // nw)))
        k = _logint(rng, 1, max(1, min(128, 16 * 64 * 2129373 // (nw * states))))
        return {"kind": kind, "r": r, "states": states, "k": k}
    if kind == "frobenius":
        r = _logint(rng, 40001, R_DEEP) | 1
        nw = (r + 63) // 64
        return {"kind": kind, "r": r, "states": _logint(rng, 1, max(1, min(64, 8 * 2129373 // nw))),
                "k": _logint(rng, 8, 96)}
    if kind == "stage2":
        r = _logint(rng, 4001, R_DEEP) | 1
        return {"kind": kind, "r": r, "degrees": rng.randint(1, 8 if r < 10_000_000 else 2)}
    if kind == "mul":
        return {"kind": kind, "abits": _logint(rng, 2000, 130_000_000),
                "bbits": _logint(rng, 2000, 130_000_000)}
    if kind == "mulbatch":
        lo = rng.uniform(12.0, 20.0)
        return {"kind": kind, "jobs": rng.randint(3, 48), "lo": lo,
                "hi": rng.uniform(lo + 1.0, 26.0), "sizes": rng.randint(2, 10**6)}
    if kind == "fft":
        return {"kind": kind, "m": rng.choice([m for m in range(8, 25) if m != 20])}
    if kind == "gcd":
        return {"kind": kind, "bits": _logint(rng, 550_000, 1_000_000), "pairs": rng.randint(1, 8),
                "common": rng.randint(1, 3000)}
    k0 = rng.randint(12, 16)
    return {"kind": "scan", "r": _sieve_prime(_logint(rng, 4400, 90_000), k0),
            "ns": rng.randint(3, 24), "k0": k0, "maxd": k0 + rng.randint(40, 120),
            "L0": 64, "block": rng.choice([1, 1, 8, 16])}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _random_poly(bits, gen):
    """A uniformly random polynomial of exactly `bits` coefficients, as words."""
    nw = (bits + 63) // 64
    t = torch.randint(-(1 << 63), (1 << 63) - 1, (nw,), dtype=torch.int64, device=DEV,
                      generator=gen)
    top = (bits - 1) % 64
    if top != 63:
        t[-1] &= (1 << (top + 1)) - 1
    t[-1] |= -(1 << 63) if top == 63 else 1 << top
    return t


def _s_values(r, n, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(1, (r - 1) // 2 + 1, size=n, dtype=np.int64)


def _batch_sizes(case):
    return W.mul_config(case["sizes"], case["jobs"], case["lo"], case["hi"])["sizes"]


def _words(n):
    return torch.zeros(int(n), dtype=torch.int64, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    st = {"case": case}
    if kind == "sieve":
        # sieve keys depend on r and s alone: a seed gives a preloaded best[]
        # (earlier results of some s), which the call extends
        rng = np.random.default_rng(seed)
        smax = case["smax"]
        pre = torch.full((smax + 1,), -1, dtype=torch.int64, device=DEV)
        known = torch.from_numpy(rng.integers(1, smax + 1, size=max(1, smax // 1000))).to(DEV)
        pre[known] = (1 << 48) | 3
        st.update(pre=pre, best=torch.empty_like(pre), ws=E.SieveWorkspace(case["dmax"]))
    elif kind == "square":
        r, n = case["r"], case["states"]
        nw = (r + 63) // 64
        stride = nw + (nw & 1)
        t = torch.randint(-(1 << 63), (1 << 63) - 1, (n, stride), dtype=torch.int64, device=DEV,
                          generator=gen)
        t[:, nw:] = 0
        if r % 64:
            t[:, nw - 1] &= (1 << (r % 64)) - 1
        st.update(x=t, scratch=torch.empty_like(t), stride=stride, nw=nw,
                  s=torch.from_numpy(_s_values(r, n, seed)).to(DEV))
    elif kind == "frobenius":
        nw = (case["r"] + 63) // 64
        out = torch.empty((case["states"], nw), dtype=torch.int64).pin_memory()
        st.update(s=_s_values(case["r"], case["states"], seed).astype(np.uint64), out=out,
                  view=out.numpy().view(np.uint64))
    elif kind == "stage2":
        G = E.TrinGPU()
        G.init(case["r"])
        G.set_s(int(_s_values(case["r"], 1, seed)[0]))
        st.update(G=G, start=_random_poly(case["r"], gen).cpu().numpy().view(np.uint64))
        G.write("A", st["start"])
        G.reset_acc()
    elif kind == "mul":
        F = E.CudaFFT()
        F.init(E.fft_m_for(case["abits"], case["bbits"]))
        st.update(F=F, a=_random_poly(case["abits"], gen), b=_random_poly(case["bbits"], gen),
                  out=_words(E.mul_out_words(case["abits"], case["bbits"])),
                  fa=_words(1 << F.m), fb=_words(1 << F.m))
    elif kind == "mulbatch":
        sizes = _batch_sizes(case)
        st["jobs"] = [(_random_poly(a, gen), a, _random_poly(b, gen), b,
                       _words(E.mul_out_words(a, b))) for a, b in sizes]
        st["ws"] = E.DeviceBuffer(E.mul_batch_workspace_bytes(sizes))
    elif kind == "fft":
        F = E.CudaFFT()
        F.init(case["m"])
        shape = (1 << case["m"],)
        st.update(F=F, **{k: torch.randint(-(1 << 63), (1 << 63) - 1, shape, dtype=torch.int64,
                                           device=DEV, generator=gen) for k in ("f", "g")})
    elif kind == "gcd":
        # pairs with a planted common factor: c * a', c * b'
        pairs = []
        c = _random_poly(case["common"], gen)
        for _ in range(case["pairs"]):
            ab = []
            for bits in (case["bits"], case["bits"] - 1):
                q = _random_poly(bits - case["common"] + 1, gen)
                out = _words(E.mul_out_words(case["common"], bits - case["common"] + 1))
                E.mul_batch_dev([(q, bits - case["common"] + 1, c, case["common"], out)])
                torch.cuda.synchronize()
                ab += [out, bits]
            pairs.append(tuple(ab))
        st["pairs"] = pairs
    else:
        r, k0 = case["r"], case["k0"]
        best = E.run_sieve(r, k0, (r - 1) // 2)
        alive = np.nonzero(best == E.U64_MAX)[0]
        alive = alive[alive >= 3]
        rng = np.random.default_rng(seed)
        st["s"] = np.sort(rng.choice(alive, size=min(case["ns"], alive.size), replace=False))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "sieve":
        st["best"].copy_(st["pre"])
        E.sieve_device(case["r"], case["dmax"], case["smax"], st["best"], dmin=case["dmin"],
                       fill=False, workspace=st["ws"])
        return st["best"]
    if kind == "square":
        E.trin_square_batch(st["x"], st["scratch"], st["stride"], case["states"], case["r"],
                            st["s"], case["k"])
        return st["x"][:, : st["nw"]]
    if kind == "frobenius":
        E.frobenius_host(case["r"], st["s"], case["k"], out=st["view"])
        return st["out"]
    if kind == "stage2":
        G = st["G"]
        for _ in range(case["degrees"]):
            G.square_A()
            G.accumulate()
        return {"F": _view(G, G.dA, G.nw), "ACC": _view(G, G.dACC, G.nw)}
    if kind == "mul":
        E.gf2x_fft_mul_dev(st["F"], st["a"], case["abits"], st["b"], case["bbits"], st["out"],
                           st["fa"], st["fb"])
        return st["out"]
    if kind == "mulbatch":
        E.mul_batch_dev(st["jobs"], workspace=st["ws"])
        return [j[4] for j in st["jobs"]]
    if kind == "fft":
        st["F"].fwd(st["f"])
        st["F"].inv(st["g"])
        return [st["f"], st["g"]]
    if kind == "gcd":
        cap = (case["common"] + 63) // 64 + 2
        degs, gs, _ = E.gcd_large(st["pairs"], g_cap_words=cap, max_parallel=64)
        return [degs] + [g.view(np.int64) for g in gs if g is not None]
    lines = E.scan(case["r"], st["s"], case["k0"], case["maxd"], L0=case["L0"], batch=32,
                   block=case["block"])
    return _lines(lines, case["maxd"])


class _DeviceWords:
    """A context's own device words, for torch to look at without a copy.
    torch keeps this object as long as the tensor, and it the context."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<i8",
                                         "data": (int(ptr), False), "version": 3}


def _view(owner, ptr, n):
    t = torch.as_tensor(_DeviceWords(owner, ptr, n), device=DEV)
    t.owner = owner
    return t


def _lines(lines, maxd):
    """Result lines as numbers: per s (s, kind, d or interval), and its factor's words."""
    rows = np.zeros((len(lines), 4), dtype=np.int64)
    masks = np.zeros((len(lines), maxd // 32 + 1), dtype=np.int64)
    for i, line in enumerate(lines):
        f = line.split()
        if f[1] == "u":
            rows[i] = (int(f[0]), 2, 0, 0)
        elif f[1].startswith("r"):
            lo, hi = f[1][1:].split("-")
            rows[i] = (int(f[0]), 3, int(lo), int(hi))
        else:
            rows[i] = (int(f[0]), 1, int(f[1]), 0)
            v = int(f[2][1:], 16)
            for w in range(masks.shape[1]):
                masks[i, w] = (v >> (32 * w)) & 0xFFFFFFFF
    return [rows, masks]


def work(case):
    """Bytes every input is read and every output written with, and whole-word
    operations that the known algorithms need at least."""
    kind = case["kind"]
    if kind == "sieve":
        # best[] read and written; one table lookup for each coset of the
        # exponents, 2^d / d of them a degree
        cosets = sum((1 << d) // d for d in range(case["dmin"], case["dmax"] + 1))
        return {"bytes": 16 * (case["smax"] + 1) + 4 * cosets, "flops": cosets}
    if kind in ("square", "frobenius"):
        # states in and out once; a squaring writes every word
        words = case["states"] * ((case["r"] + 63) // 64)
        return {"bytes": 8 * words * (2 if kind == "square" else 1), "flops": words * case["k"]}
    if kind == "stage2":
        nw = (case["r"] + 63) // 64
        return {"bytes": 32 * nw,
                "flops": case["degrees"] * (nw + _mul_ops(case["r"], case["r"]))}
    if kind == "mul":
        ab, bb = case["abits"], case["bbits"]
        return {"bytes": (ab + bb) // 4, "flops": _mul_ops(ab, bb)}
    if kind == "mulbatch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(a + b for a, b in sizes) // 4,
                "flops": sum(_mul_ops(a, b) for a, b in sizes)}
    if kind == "fft":
        n = 1 << case["m"]
        return {"bytes": 32 * n, "flops": 2 * n * case["m"]}
    if kind == "gcd":
        # operands in; about log2(words) products of the operands' size
        bits = case["bits"]
        lg = max(1, (bits // 64).bit_length())
        return {"bytes": case["pairs"] * bits // 4,
                "flops": case["pairs"] * lg * _mul_ops(bits // 2, bits // 2)}
    nw = (case["r"] + 63) // 64
    deg = case["maxd"] - case["k0"]
    return {"bytes": 8 * nw * case["ns"],
            "flops": case["ns"] * deg * (nw + _mul_ops(case["r"], case["r"]) // case["block"])}


def _mul_ops(abits, bbits):
    """One operation a point and level of the three transforms of a product."""
    m = max(1, ((abits + bbits) // 32).bit_length())
    return 3 * m * ((abits + bbits) // 32 + 1)


def exact(case, seed):
    """Bit strings and whole numbers only: nothing is rounded, so there is no
    value in 64 bits to be nearer to."""
    return None
