"""What the performance of this framework is measured on: the prover's work through the public Python API.

A case is one of six kinds.  `msm`: one multi-scalar multiplication, its inputs on the device or in host arrays
(msm_best).  `commit`: the commitments of a phase, many MSMs of mixed sizes in one call over a resident SRS, stored
as a fixed-base window table or plain.  `ntt`: one EvaluationDomain transform, alone or for several polynomials of a
domain.  `quotient`: h(X) on the extended coset of the standard circuit.  `products`: the permutation product and the
logup columns.  `proofs`: create_proof for one or more requests of one key.

Results are elements of finite fields, points and proof bytes: exact, and compared bit by bit.
"""
import random

import numpy as np
import torch

from _loader import load

mzk = load()

# r's top 64-bit limb: an element whose top limb lies below it is below r
FR_TOP = 0x73EDA753299D7D48
FR_ONE = (0x00000001FFFFFFFE, 0x5884B7FA00034802, 0x998C4FEFECBC4FF5, 0x1824B159ACC5056F)  # Montgomery one
DEGREE = 5            # the standard circuit's constraint degree: extended domain of 4 n rows
BLINDING = 7          # its blinding factors
# 32-bit multiply-adds of one Montgomery product (two halves of 2 s^2 + s partial products)
FP_MUL, FR_MUL = 600, 272
QUOTIENT_FR_MULS = 37  # per extended row of the standard circuit

_ctx = None


def context():
    """The program's one device context."""
    global _ctx
    if _ctx is None:
        _ctx = mzk.Context(0)
    return _ctx


class Column:
    """A torch tensor of field elements or points as the API's device buffer."""

    def __init__(self, tensor):
        self.tensor, self.ptr = tensor, tensor.data_ptr()


# ---- cases -------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest commitments (small circuits, verifier-side MSMs): launches and latency
        {"name": "msm 1k", "kind": "msm", "n": 1000, "host": False, "sparse": False},
        # a commitment issued from host memory, as a caller of the reference's msm_best does
        {"name": "msm 64k host", "kind": "msm", "n": 1 << 16, "host": True, "sparse": False},
        # an ordinary polynomial's commitment, length not a power of two
        {"name": "msm 1M ragged", "kind": "msm", "n": 1000003, "host": False, "sparse": False},
        # the largest commitment
        {"name": "msm 16M", "kind": "msm", "n": 1 << 24, "host": False, "sparse": False},
        # the commitments of mixed circuits in one call over the prover's window table, one in four sparse
        {"name": "commit table", "kind": "commit", "items": 24, "log_min": 12, "log_max": 20, "sizes": 7, "table": True},
        # a small circuit's single transform
        {"name": "ntt 4k", "kind": "ntt", "op": "coeff_to_lagrange", "k": 12, "count": 1},
        # the witness polynomials of a proof to the extended coset
        {"name": "ntt extended k18 x7", "kind": "ntt", "op": "coeff_to_extended", "k": 18, "count": 7},
        # the largest inverse transform: h(X) of a circuit of 2^22 rows back to coefficients
        {"name": "ntt inverse 16M", "kind": "ntt", "op": "extended_to_coeff", "k": 22, "count": 1},
        # the quotient of an ordinary circuit
        {"name": "quotient k18", "kind": "quotient", "k": 18},
        # the grand products of an ordinary circuit
        {"name": "products k17", "kind": "products", "k": 17},
        # one proof of a small circuit: the latency of a request served alone
        {"name": "proof k14", "kind": "proofs", "k": 14, "count": 1},
        # a served wave of proofs
        {"name": "proofs k16 x8", "kind": "proofs", "k": 16, "count": 8},
    ]


def draw(rng):
    def spread(lo, hi):  # log-uniform whole number
        return int(round(2 ** rng.uniform(np.log2(lo), np.log2(hi))))

    kind = rng.choice(["msm", "msm", "commit", "ntt", "ntt", "quotient", "products", "proofs", "proofs"])
    if kind == "msm":
        host = rng.random() < 0.3
        n = spread(300, (1 << 20) if host else (1 << 23))
        return {"kind": kind, "n": n | 1 if rng.random() < 0.5 else n, "host": host, "sparse": rng.random() < 0.25}
    if kind == "commit":
        return {"kind": kind, "items": rng.randint(2, 32), "log_min": rng.randint(10, 14),
                "log_max": rng.randint(15, 20), "sizes": rng.randint(0, 1 << 20), "table": rng.random() < 0.7}
    if kind == "ntt":
        op = rng.choice(["coeff_to_lagrange", "lagrange_to_coeff", "coeff_to_extended", "extended_to_coeff"])
        k = rng.randint(8, 22)
        return {"kind": kind, "op": op, "k": k, "count": spread(1, max(1, min(24, (1 << 22) >> k)))}
    if kind == "quotient":
        return {"kind": kind, "k": rng.randint(10, 19)}
    if kind == "products":
        return {"kind": kind, "k": rng.randint(10, 20)}
    k = rng.randint(10, 18)
    return {"kind": kind, "k": k, "count": rng.randint(1, max(1, min(12, (1 << 19) >> k)))}


# ---- inputs ------------------------------------------------------------------------------------------------------

def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def elements(gen, n, sparse=False):
    """n field elements (Montgomery), uniform; sparse: 90 % of them zero or one, as in selector columns."""
    full = (-(1 << 63), (1 << 63) - 1)
    a = torch.randint(*full, (n, 4), generator=gen, device="cuda", dtype=torch.int64)
    a[:, 3] = torch.randint(0, FR_TOP, (n,), generator=gen, device="cuda", dtype=torch.int64)
    if sparse:
        u = torch.rand(n, generator=gen, device="cuda")
        a[u < 0.9] = torch.tensor(np.array(FR_ONE, np.uint64).view(np.int64), device="cuda")
        a[u < 0.45] = 0
    return a


def points(seed, n):
    """n points of the group, [r_i] G."""
    p = torch.empty((n, 12), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    context().gen_bases(seed, n, out=Column(p))
    return p


def challenge(rng):
    return np.array([rng.getrandbits(64) for _ in range(3)] + [rng.randrange(FR_TOP)], np.uint64)


def commit_sizes(case):
    rng = random.Random(case["sizes"])
    return [int(2 ** rng.uniform(case["log_min"], case["log_max"])) for _ in range(case["items"])]


def proving_key(k, seed):
    """A circuit instance with its domain and its SRS (over the window table that the library advises)."""
    ctx, n = context(), 1 << k
    domain = mzk.EvaluationDomain(ctx, DEGREE, k)
    c = mzk.prover_table_width(k)
    rows = ctx.msm_table_rows(c)
    srs = torch.empty((rows * 4 * n, 12), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    at = srs.data_ptr()
    secret = challenge(random.Random(seed))
    domain.srs_setup_device(secret, at, at + n * 96, at + 2 * n * 96, at + 3 * n * 96)
    ctx.msm_window_table(at, 4 * n, c, rows)
    desc = mzk.SrsDesc(at, 4 * n, 0, n, 2 * n, 3 * n, c, rows, n)
    return mzk.Config3Instance(ctx, domain, desc, seed), srs


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    gen, rng = generator(seed), random.Random(seed)
    if kind == "msm":
        scalars, bases = elements(gen, case["n"], case["sparse"]), points(seed, case["n"])
        if case["host"]:
            return {"case": case, "scalars": scalars.cpu().numpy().view(np.uint64),
                    "bases": bases.cpu().numpy().view(np.uint64)}
        torch.cuda.synchronize()
        return {"case": case, "scalars": Column(scalars), "bases": Column(bases)}
    if kind == "commit":
        sizes = commit_sizes(case)
        length = max(sizes)
        c = mzk.prover_table_width((length - 1).bit_length()) if case["table"] else 0
        rows = ctx.msm_table_rows(c) if c else 1
        table = torch.empty((rows * length, 12), dtype=torch.int64, device="cuda")
        table[:length] = points(seed, length)
        scalars = [Column(elements(gen, n, i % 4 == 3)) for i, n in enumerate(sizes)]
        torch.cuda.synchronize()
        if c:
            ctx.msm_window_table(table.data_ptr(), length, c, rows)
        return {"case": case, "table": Column(table), "length": length, "c": c, "rows": rows,
                "items": [(s.ptr, 0, n) for s, n in zip(scalars, sizes)], "scalars": scalars}
    if kind == "ntt":
        domain = mzk.EvaluationDomain(ctx, DEGREE, case["k"])
        n, extended = domain.n, domain.extended_len
        n_in = extended if case["op"] == "extended_to_coeff" else n
        n_out = extended if "extended" in case["op"] else n
        ins = [Column(elements(gen, n_in)) for _ in range(case["count"])]
        outs = [Column(torch.empty((n_out, 4), dtype=torch.int64, device="cuda")) for _ in range(case["count"])]
        torch.cuda.synchronize()
        return {"case": case, "domain": domain, "ins": ins, "outs": outs}
    if kind == "quotient":
        domain = mzk.EvaluationDomain(ctx, DEGREE, case["k"])
        rows = domain.extended_len

        def some(count):
            return [Column(elements(gen, rows)) for _ in range(count)]

        cols = {"advice": some(3), "fixed": some(7), "gate_fixed": [0, 1, 2, 3, 4], "gate_advice": [0, 1, 2],
                "perm_cols": [(0, 0), (0, 1), (0, 2)], "perm_sigma": some(3), "perm_z": some(1), "chunk_len": 3,
                "blinding_factors": BLINDING,
                "lookup": dict(zip("hzm", some(3)), input=0, table=5, selector=6)}
        cols["l0"], cols["l_last"], cols["l_active"] = some(3)
        for name in ("y", "beta", "gamma", "theta"):
            cols[name] = challenge(rng)
        out = Column(torch.empty((rows, 4), dtype=torch.int64, device="cuda"))
        torch.cuda.synchronize()
        desc = mzk.build_quotient_desc(cols, case["k"], domain.extended_k, lambda c: c.ptr)
        return {"case": case, "domain": domain, "desc": desc, "columns": cols, "out": out}
    if kind == "products":
        domain = mzk.EvaluationDomain(ctx, DEGREE, case["k"])
        ins = [Column(elements(gen, domain.n, i == 7)) for i in range(9)]
        outs = [Column(torch.empty((domain.n, 4), dtype=torch.int64, device="cuda")) for _ in range(3)]
        torch.cuda.synchronize()
        return {"case": case, "domain": domain, "ins": ins, "outs": outs, "beta": challenge(rng),
                "gamma": challenge(rng), "blinds": np.stack([challenge(rng) for _ in range(2 * BLINDING)])}
    instance, srs = proving_key(case["k"], seed)
    jobs = [(instance.key, instance.witness(seed + 2 * i), instance.blinds(seed + 2 * i + 1))
            for i in range(case["count"])]
    return {"case": case, "instance": instance, "srs": srs, "jobs": jobs}


# ---- one pass ----------------------------------------------------------------------------------------------------

def run(state):
    ctx, case = context(), state["case"]
    kind = case["kind"]
    if kind == "msm":
        if case["host"]:
            return ctx.msm_best(state["scalars"], state["bases"])
        return ctx.msm_device(state["scalars"], state["bases"], case["n"])
    if kind == "commit":
        if state["c"]:
            return ctx.msm_batch_table_device(state["table"], state["length"], state["c"], state["rows"],
                                              min(n for _, _, n in state["items"]), state["items"])
        return ctx.msm_batch_device(state["table"].ptr, state["length"], state["items"])
    if kind == "ntt":
        ins, outs = state["ins"], state["outs"]
        if case["count"] == 1:
            state["domain"].op_device(case["op"], ins[0].ptr, outs[0].ptr)
        else:
            state["domain"].op_batch_device(case["op"], [c.ptr for c in ins], [c.ptr for c in outs])
        return [c.tensor for c in outs]
    if kind == "quotient":
        state["domain"].quotient_eval_device(state["desc"], state["out"].ptr)
        return state["out"].tensor
    if kind == "products":
        a, z, h, agg = state["ins"], *state["outs"]
        domain, blinds = state["domain"], state["blinds"]
        domain.permutation_z_device(a[:3], a[3:6], 3, BLINDING, blinds[:BLINDING], state["beta"], state["gamma"], [z])
        domain.logup_device([[a[0]]], a[6], a[7], a[8], BLINDING, blinds[BLINDING:], state["beta"], [h], agg)
        return [c.tensor for c in (z, h, agg)]
    return [np.frombuffer(p, np.uint8) for p in mzk.create_proofs(ctx, state["jobs"])]


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def msm_muls(n, windows):
    """Fp products of an MSM: a mixed addition (10) per point and window, the bucket sums left out."""
    return 10 * n * windows


def fft_muls(n):
    return n // 2 * (n.bit_length() - 1)


def work(case):
    kind = case["kind"]
    if kind == "msm":
        n = case["n"]
        share = 0.1 if case["sparse"] else 1.0
        windows = -(-255 // mzk.msm_pick_window(n))
        return {"bytes": 128 * n, "flops": 2 * FP_MUL * share * msm_muls(n, windows)}
    if kind == "commit":
        sizes = commit_sizes(case)
        c = mzk.prover_table_width((max(sizes) - 1).bit_length()) if case["table"] else 0
        muls = sum((0.1 if i % 4 == 3 else 1.0) * msm_muls(n, -(-255 // (c or mzk.msm_pick_window(n))))
                   for i, n in enumerate(sizes))
        return {"bytes": 32 * sum(sizes) + 96 * max(sizes), "flops": 2 * FP_MUL * muls}
    n = 1 << case["k"]
    if kind == "ntt":
        extended = "extended" in case["op"]
        size, n_in = (4 * n if extended else n), (4 * n if case["op"] == "extended_to_coeff" else n)
        return {"bytes": 32 * case["count"] * (n_in + size), "flops": 2 * FR_MUL * case["count"] * fft_muls(size)}
    if kind == "quotient":
        return {"bytes": 32 * 4 * n * 21, "flops": 2 * FR_MUL * QUOTIENT_FR_MULS * 4 * n}
    if kind == "products":
        return {"bytes": 32 * n * 12, "flops": 2 * FR_MUL * 30 * n}
    # a proof of the standard circuit: 13 commitments of n points, seven witness columns to coefficients and to the
    # extended coset, the quotient, and h back; its columns and SRS read once
    c = mzk.prover_table_width(case["k"])
    muls = FP_MUL * 13 * msm_muls(n, -(-255 // c))
    muls += FR_MUL * (7 * (fft_muls(n) + fft_muls(4 * n)) + fft_muls(4 * n) + QUOTIENT_FR_MULS * 4 * n)
    return {"bytes": 32 * n * case["count"] * 3 + 96 * 4 * n + 32 * 4 * n * 13, "flops": 2 * case["count"] * muls}


def exact(case, seed):
    """Every output is an exact field element, point or byte, held to equality: none is rounded."""
    return None
