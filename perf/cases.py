"""The work that programs have this library do, as cases that can be timed and compared.

Every case goes through the package's public entry points on inputs made on
the GPU from a seed: whole proofs of the benchmark circuit, and the parts of a
proof that a prover calls by themselves (commitments over plain bases and over
window tables, transforms, batch inversion, the quotient, the lookup and
permutation arguments, the opening).  Results are residues and curve points in
canonical form, so every output is compared exactly.
"""
import importlib
import importlib.util
import os
import sys

import numpy as np
import torch

R = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001     # the scalar field's order
Q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47     # the base field's order
MONT = 1 << 256
ZETA = 0x30644E72E131A029048B6E193FD84104CC37A73FEC2BC5E9B8CA0B2D36636F23   # the coset generator
# operations of one 256-bit Montgomery product: 8 x 8 word products for a b, as many for the reduction,
# 8 quotient words, each a multiply and an add
PRODUCT = 2 * (64 + 64 + 8)


def _pkg():
    name = "halo2_gpu_b200"
    if name not in sys.modules:
        root = os.path.join(os.getcwd(), "halo2-gpu_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _sub(name):
    return importlib.import_module(_pkg().__name__ + "." + name)


# --- the cases ---------------------------------------------------------------------

def listed():
    return [
        # a whole proof of the serving stream's most frequent size, transcript included
        {"name": "proof_k16", "kind": "proof", "k": 16},
        # a whole proof of its largest size: the step that production time goes into
        {"name": "proof_k22", "kind": "proof", "k": 22},
        # the headline kernel: one commitment of 2^22 witness-like scalars over plain bases, all on the device
        {"name": "msm_k22_witness", "kind": "msm", "n": 1 << 22, "mix": 1, "host": False},
        # a commitment whose scalars are still on the host, at the size that the CPU path is compared at
        {"name": "msm_k16_host", "kind": "msm", "n": 1 << 16, "mix": 0, "host": True},
        # a small circuit's commitment, odd length: latency and launches
        {"name": "msm_1000", "kind": "msm", "n": 1000, "mix": 0, "host": False},
        # the advice commitments of one proof over a resident window table, as one batch
        {"name": "commit_4x_k18", "kind": "commit", "k": 18, "n": 1 << 18, "jobs": 4, "mix": 1},
        # lagrange_to_coeff of one small proof's ten columns
        {"name": "ifft_10x_k16", "kind": "ntt", "type": 2, "k": 16, "count": 10},
        # the coset extension 2^22 -> 2^24 of one full-size polynomial
        {"name": "coset_ext_k22", "kind": "ntt", "type": 3, "k": 22, "count": 1},
        # the inversion of a full-size column set's denominators
        {"name": "invert_k24", "kind": "invert", "n": 1 << 24, "zeros": False},
        # one extended part of the quotient: gates, permutation and lookup in one pass
        {"name": "quotient_k20", "kind": "quotient", "k": 20},
        # the lookup's permuted columns and the three grand products of one proof
        {"name": "arguments_k20", "kind": "arguments", "k": 20},
        # the opening of one mid-size proof: 24 evaluations, two commitments, the divisions between them
        {"name": "opening_k18", "kind": "opening", "k": 18},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["proof", "msm", "msm", "commit", "ntt", "ntt", "invert", "quotient", "arguments", "opening"])
    if kind == "proof":
        return {"kind": kind, "k": rng.randint(10, 20)}
    if kind == "msm":
        return {"kind": kind, "n": _log_int(rng, 33, 1 << 22), "mix": rng.randint(0, 1), "host": rng.random() < 0.4}
    if kind == "commit":
        k = rng.randint(10, 20)
        return {"kind": kind, "k": k, "n": _log_int(rng, (1 << k) // 16, 1 << k), "jobs": rng.randint(1, 7),
                "mix": rng.randint(0, 1)}
    if kind == "ntt":
        t = rng.choice([1, 2, 3, 6])
        k = rng.randint(6, 22 if t != 3 else 21)
        return {"kind": kind, "type": t, "k": k, "count": rng.randint(1, max(1, min(16, (1 << 23) >> k)))}
    if kind == "invert":
        return {"kind": kind, "n": _log_int(rng, 17, 1 << 24), "zeros": rng.random() < 0.5}
    return {"kind": kind, "k": rng.randint(10, 20)}


# --- inputs -------------------------------------------------------------------------

def _uniform(n, seed):
    """n residues below 2^253 as Montgomery images, from torch's generator."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + 17)
    v = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    v[:, 3] &= (1 << 61) - 1
    return v.view(torch.uint8).reshape(-1)


def _scalars(n, seed, mix):
    """Uniform scalars, or a witness column's: half uniform, 30% below 2^64, 20% zeros and ones."""
    return _uniform(n, seed) if not mix else _pkg().random_fr_device(n, seed, 1)


def _tau(seed):
    return (0xABCDEF12345 + 7919 * seed) % R


def _ints(t):
    a = t.cpu().numpy().view("<u8").reshape(-1, 4).tolist()
    inv = pow(MONT, -1, R)
    return [(x[0] | x[1] << 64 | x[2] << 128 | x[3] << 192) * inv % R for x in a]


def _bytes_of(xs, m=R):
    return np.frombuffer(b"".join((x * MONT % m).to_bytes(32, "little") for x in xs), np.uint8)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_proof(case, seed):
    """The resident SRS, its tables and the key of one circuit size: what a proving service holds."""
    res = _sub("prover").Resident(_pkg(), case["k"], seed=_tau(seed))
    res.lagrange_table(case["k"])
    res.key_cosets(case["k"])
    res.verifying_key(case["k"])
    return {"kind": "proof", "res": res, "k": case["k"], "seed": seed + 1, "stream": torch.cuda.current_stream()}


def _prepare_msm(case, seed):
    h, n = _pkg(), case["n"]
    sc = _scalars(n, seed, case["mix"])
    s = {"kind": "msm", "n": n, "host": case["host"], "bases": h.srs_device(_tau(seed), n)}
    if case["host"]:
        s["scalars"] = sc.cpu().numpy().view(np.uint64).reshape(n, 4)
    else:
        s["scalars"], s["ws"], s["out"] = sc, h.msm_workspace(n), h.dev_empty(96)
    return s


def _prepare_commit(case, seed):
    h, tn, n, jobs = _pkg(), 1 << case["k"], case["n"], case["jobs"]
    table = h.msm_table_precompute(h.srs_device(_tau(seed), tn), tn)
    sc = [_scalars(n, seed * 16 + i, case["mix"]) for i in range(jobs)]
    outs = [h.dev_empty(96) for _ in range(jobs)]
    js = h.msm_batch_jobs(sc, [table] * jobs, outs, [n] * jobs, table_n=tn)
    return {"kind": "commit", "jobs": js, "count": jobs, "ws": h.msm_batch_workspace(js, jobs, jobs), "outs": outs,
            "keep": (table, sc)}


def _prepare_ntt(case, seed):
    h, t, k = _pkg(), case["type"], case["k"]
    dom = _sub("fields").EvaluationDomain(4, k)
    ek = dom.extended_k if t == 3 else k
    omega = {1: dom.omega, 2: dom.omega_inv, 3: dom.extended_omega, 6: dom.omega}[t]
    divisor = {1: 1, 2: dom.ifft_divisor, 3: 1, 6: ZETA * dom.extended_omega % R}[t]
    ins = [_uniform(1 << k, seed * 32 + i) for i in range(case["count"])]
    outs = [h.dev_empty(32 << ek) for _ in ins]
    ws = h.dev_empty(h.lib()._halo2_fft_many_to_device_workspace_size(t, k, ek))
    return {"kind": "ntt", "type": t, "k": k, "ek": ek, "ins": ins, "outs": outs, "omega": omega, "divisor": divisor,
            "ws": ws}


def _prepare_invert(case, seed):
    h, n = _pkg(), case["n"]
    x = _uniform(n, seed)
    if case["zeros"]:
        x.view(n, 32)[5::17] = 0
    return {"kind": "invert", "n": n, "x": x, "out": torch.empty_like(x),
            "ws": h.dev_empty(h.lib().h2b_batch_invert_workspace_size(n))}


def _prepare_quotient(case, seed):
    """Twenty columns' values on one coset of the extended domain (uniform, as any coset's are) and the constraint
    system's rules."""
    C, n = _sub("circuit"), 1 << case["k"]
    dom = _sub("fields").EvaluationDomain(C.DEGREE, case["k"])
    cols = [_uniform(n, seed * 32 + i) for i in range(20)]
    return {"kind": "quotient", "n": n, "dom": dom, "cols": cols, "gates": C.gate_graph(),
            "lookup": C.lookup_product_graph(), "seed": seed}


def _prepare_arguments(case, seed):
    h, C = _pkg(), _sub("circuit")
    pk = C.ProvingKey(h, case["k"])
    adv, inst, _ = C.synthesize(h, pk, seed + 1)
    F = _sub("fields")
    up = lambda v: h.to_dev(F.fr_mont_limbs([v % R]))  # noqa: E731
    beta, gamma = up(0x1234567 * (seed + 3)), up(0x89ABCDEF1 * (seed + 5))
    dws = [up(pow(F.DELTA, C.CHUNK_LEN * s, R)) for s in range(2)]
    return {"kind": "arguments", "n": pk.n, "u": pk.u, "pk": pk, "adv": adv, "inst": inst, "beta": beta,
            "gamma": gamma, "delta": up(F.DELTA), "omega": up(pk.dom.omega), "one": up(1), "dws": dws}


def _prepare_opening(case, seed):
    h, P, n = _pkg(), _sub("prover"), 1 << case["k"]
    C = _sub("circuit")
    dom = _sub("fields").EvaluationDomain(C.DEGREE, case["k"])
    names = ([f"adv{i}" for i in range(4)] + ["z0", "z1", "zl", "pa", "ps"] + [f"fixed{i}" for i in range(3)] +
             [f"sigma{i}" for i in range(4)] + ["h", "random"])
    polys = {m: _uniform(n, seed * 32 + i) for i, m in enumerate(names)}
    queries, _ = P.open_queries_for(dom, pow(7, 1000 + seed, R), polys)
    return {"kind": "opening", "n": n, "queries": queries, "table": h.msm_table_precompute(h.srs_device(_tau(seed), n), n),
            "challenges": [pow(11, 50 + 3 * seed + i, R) for i in range(3)], "keep": polys,
            "ws": h.dev_empty(h.lib().h2b_msm_table_workspace_size(n, n))}


# --- one pass -------------------------------------------------------------------------

def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_proof(s):
    w = _sub("prover").ProofWorkload(s["res"], s["k"], s["seed"], transcript=True)
    commits, evals = w.run(s["stream"])
    return {"commits": commits, "evals": evals, "proof": np.frombuffer(w.proof, np.uint8)}


def _run_msm(s):
    h = _pkg()
    if s["host"]:
        return h.multiexp_gpu_device_bases(s["scalars"], s["bases"], s["n"]).view(np.uint8)
    h.msm_device(s["scalars"], s["bases"], s["out"], s["n"], s["ws"])
    return s["out"]


def _run_commit(s):
    _pkg().msm_batch(s["jobs"], s["count"], s["count"], s["ws"])
    return s["outs"]


def _run_ntt(s):
    return _pkg().fft_many_to_device(s["type"], s["k"], s["ek"], s["ins"], s["outs"], s["omega"], s["divisor"],
                                     ws=s["ws"])


def _run_invert(s):
    """The library inverts in place, so a program that still needs the denominators inverts a copy."""
    s["out"].copy_(s["x"])
    _pkg().batch_invert_device_scratch(s["out"], s["n"], 0, s["ws"])
    return s["out"]


def _run_quotient(s):
    h, F, C = _pkg(), _sub("fields"), _sub("circuit")
    n, c, dom = s["n"], s["cols"], s["dom"]
    beta, gamma, y = (pow(5, 77 * (s["seed"] + 1) + i, R) for i in range(3))
    shift = dom.extended_omega
    g_rules, g_parts, g_consts = s["gates"]
    l_rules, l_parts, l_consts = s["lookup"]
    fx, adv, inst, sg, z, zl, pa, ps = c[0:3], c[3:7], c[7], c[8:12], c[12:14], c[14], c[15], c[16]
    perm = dict(prods=z, sigmas=sg, cols=[adv[0], adv[1], adv[2], inst], beta=beta, gamma=gamma, delta=F.DELTA,
                delta_start=beta * ZETA % R, ext_omega=shift, omega=dom.omega, chunk_len=C.CHUNK_LEN,
                last_rotation=-(C.BLINDING_FACTORS + 1), rot_scale=1, isize=n)
    look = dict(rules=(F.fr_mont_limbs([beta, gamma]), l_consts, l_rules, l_parts), z=zl, pin=pa, ptab=ps, beta=beta,
                gamma=gamma)
    out = h.dev_empty(32 * n)
    return h.quotient_fused_device(fx, [inst], adv, (np.zeros((0, 4), np.uint64), g_consts, g_rules, g_parts), y, c[17],
                                   c[18], c[19], perm, [look], n, 1, 0, n, out, 1, 0, dom.t_evaluations[1])


def _run_arguments(s):
    h, n, u, pk, adv = _pkg(), s["n"], s["u"], s["pk"], s["adv"]
    b, t = adv[1], pk.fixed_values[2]
    pa, ps = torch.zeros(32 * n, dtype=torch.uint8, device="cuda"), torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
    h.permute_expression_pair_device(b, t, pa, ps, n, u)
    cols, outs, prefix = [adv[0], adv[1], adv[2], s["inst"]], [pa, ps], s["one"]
    for i in range(2):
        mod = h.dev_empty(32 * n)
        h.call("_halo2_poly_fill_one", h.ptr(mod), n, h.stream_handle())
        dw = s["dws"][i].clone()                        # the entry point advances it
        h.permutation_product_device(mod, pk.sigma_values[2 * i:2 * i + 2], cols[2 * i:2 * i + 2], s["beta"],
                                     s["gamma"], s["delta"], s["omega"], dw, u)
        z = torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
        z[:32] = prefix
        z[32:32 * (u + 1)] = mod[:32 * u]
        h.grand_product_device(z, prefix, u, offset=1)
        prefix = z[32 * u:32 * (u + 1)]
        outs.append(z)
    ratio, zl = h.dev_empty(32 * n), torch.zeros(32 * n, dtype=torch.uint8, device="cuda")
    h.lookup_product_device(ratio, pa, ps, b, t, s["beta"], s["gamma"], u)
    zl[:32] = s["one"]
    zl[32:32 * (u + 1)] = ratio[:32 * u]
    h.grand_product_device(zl, s["one"], u, offset=1)
    return outs + [zl]


def _run_opening(s):
    h = _pkg()

    def commit(d):
        return h.msm_device_table(d, s["table"], s["n"], h.dev_empty(96), s["n"], ws=s["ws"])

    evals, points, at_u = _sub("shplonk").open_queries(h, s["queries"], iter(s["challenges"]), commit)
    return {"evals": _bytes_of(evals), "points": points, "at_u": int(at_u)}


# --- what a pass cannot do without ------------------------------------------------------

def _msm_work(n, resident_slices=1):
    """16 additions a point (16-bit windows over 254 bits) of 6 products each (affine, the inversions shared)."""
    return 96 * n, 16 * 6 * n * PRODUCT


def work(case):
    kind = case["kind"]
    if kind == "msm":
        b, f = _msm_work(case["n"])
    elif kind == "commit":
        b, f = (case["jobs"] * x for x in _msm_work(case["n"]))
    elif kind == "ntt":
        ek = case["k"] + (2 if case["type"] == 3 else 0)
        b = case["count"] * (32 * (1 << case["k"]) + 32 * (1 << ek))
        f = case["count"] * (1 << ek) * ek // 2 * PRODUCT
    elif kind == "invert":
        b, f = 64 * case["n"], 3 * case["n"] * PRODUCT
    elif kind == "quotient":
        b, f = 21 * 32 << case["k"], (54 << case["k"]) * PRODUCT
    elif kind == "arguments":
        # b, t, four columns, four sigmas in; two permuted columns and three products out; about 22 products a row
        b, f = 15 * 32 << case["k"], (22 << case["k"]) * PRODUCT
    elif kind == "opening":
        # 16 polynomials read for the evaluations and again for each combination; two commitments
        n = 1 << case["k"]
        mb, mf = _msm_work(n)
        b, f = 3 * 16 * 32 * n + 2 * mb, (24 + 32 + 24) * n * PRODUCT + 2 * mf
    else:
        # 14 commitments, ten inverse transforms, four parts of ten transforms and a quotient, the inverse extended
        # transform, the arguments and the opening's polynomial work
        n, k = 1 << case["k"], case["k"]
        mb, mf = _msm_work(n)
        b = 14 * mb + (10 * 64 + 4 * 10 * 64 + 4 * 21 * 32 + 4 * 64 + 15 * 32 + 3 * 16 * 32) * n
        f = 14 * mf + (50 * n * k // 2 + 4 * n * (k + 2) // 2 + 4 * 54 * n + 22 * n + 80 * n) * PRODUCT
    return {"bytes": int(b), "flops": int(f)}


def tolerance(case):
    return "exact"


# --- the same by Python's integers --------------------------------------------------------

def _g1_add(a, b):
    if a is None or b is None:
        return b if a is None else a
    (x1, y1), (x2, y2) = a, b
    if x1 == x2:
        if (y1 + y2) % Q == 0:
            return None
        m = 3 * x1 * x1 * pow(2 * y1, -1, Q) % Q
    else:
        m = (y2 - y1) * pow(x2 - x1, -1, Q) % Q
    x = (m * m - x1 - x2) % Q
    return x, (m * (x1 - x) - y1) % Q


def _commitment(scalars, tau):
    """[sum_i s_i tau^i] G as the 96-byte image {x, y, 1}, or {0, 1, 0}."""
    e = 0
    for s in reversed(scalars):
        e = (e * tau + s) % R
    acc, p = None, (1, 2)
    while e:
        acc = _g1_add(acc, p) if e & 1 else acc
        p = _g1_add(p, p)
        e >>= 1
    return _bytes_of([0, 1, 0] if acc is None else [acc[0], acc[1], 1], Q)


def _root(k):
    return pow(pow(7, (R - 1) >> 28, R), 1 << (28 - k), R)


def _dft(a, w):
    n, k = len(a), len(a).bit_length() - 1
    a = [a[int(format(i, "0%db" % k)[::-1], 2)] for i in range(n)]
    m = 1
    while m < n:
        step, ws = pow(w, n // (2 * m), R), [1]
        for _ in range(m - 1):
            ws.append(ws[-1] * step % R)
        for i in range(0, n, 2 * m):
            for j in range(m):
                u, v = a[i + j], a[i + j + m] * ws[j] % R
                a[i + j], a[i + j + m] = (u + v) % R, (u - v) % R
        m *= 2
    return a


def exact(case, seed):
    kind = case["kind"]
    if kind == "msm" and not case["mix"] and case["n"] <= 1 << 18:
        return _commitment(_ints(_uniform(case["n"], seed)), _tau(seed))
    if kind == "commit" and not case["mix"] and case["n"] * case["jobs"] <= 1 << 18:
        return [_commitment(_ints(_uniform(case["n"], seed * 16 + i)), _tau(seed)) for i in range(case["jobs"])]
    if kind == "ntt" and (case["count"] * case["k"] << case["k"] + 2 * (case["type"] == 3)) <= 11 << 20:
        outs = []
        for i in range(case["count"]):
            k, t = case["k"], case["type"]
            a = _ints(_uniform(1 << k, seed * 32 + i))
            if t == 2:
                d = pow(1 << k, -1, R)
                a = [x * d % R for x in _dft(a, pow(_root(k), -1, R))]
            else:
                c = {1: 1, 3: ZETA, 6: ZETA * _root(k + 2) % R}[t]
                p = 1
                for j in range(len(a)):
                    a[j], p = a[j] * p % R, p * c % R
                a = _dft(a + [0] * (3 << k), _root(k + 2)) if t == 3 else _dft(a, _root(k))
            outs.append(_bytes_of(a))
        return outs
    if kind == "invert" and case["n"] <= 1 << 17:
        x = _uniform(case["n"], seed)
        if case["zeros"]:
            x.view(-1, 32)[5::17] = 0
        return _bytes_of([pow(v, -1, R) if v else 0 for v in _ints(x)])
    return None
