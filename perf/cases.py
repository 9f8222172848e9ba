"""The workloads whose speed is tracked: what a program built on hmpc_gb300
has it do, each through the public Python entry points, over the range of
sizes it is used at.

A case is one operation at one size.  `prepare` makes what the program holds
before the call (a queue, registered moduli with their tables and tuned
plans, keys, inputs on the device); `run` is the call itself.  Sampled
operations draw from a nonce set before the call, so a pass is reproducible.
"""
import random

import numpy as np
import torch

from hmpc_gb300 import lhe, serving
from hmpc_gb300.batch import NttBatch
from hmpc_gb300.comp import Queue, Tensor
from hmpc_gb300.moduli import MODULI

P = MODULI["p64"]
LIMBS = {name: (value.bit_length() + 31) // 32 for name, value in MODULI.items()}
CIPHERTEXT_MODULI = ["q128", "q160", "q192", "q224", "q256"]  # 4 to 8 limbs


def listed():
    return [
        # one ring element to NTT form and back: the reference's examples/ntt.cpp, the smallest call there is
        {"name": "ntt_4096", "op": "ntt", "q": "ntt", "log_n": 12, "batch": 1},
        # a key pair: two sampled transforms of one polynomial each, a uniform polynomial and their combination
        {"name": "keygen_32768", "op": "keygen", "q": "q256", "log_n": 15},
        # a client's few messages, encrypted without tuning any plan first
        {"name": "enc_3x8192", "op": "enc", "q": "q256", "log_n": 13, "batch": 3, "tuned": False, "ntt_form": False},
        # the bulk encryption of the BGV workload (bench.py): 256 messages, plans tuned once
        {"name": "enc_256x32768", "op": "enc", "q": "q256", "log_n": 15, "batch": 256, "tuned": True,
         "ntt_form": False},
        # a server's answers decrypted to NTT-form plaintexts: the inverse transform mod q, the lift to p, NTT mod p
        {"name": "dec_33x16384", "op": "dec", "q": "q192", "log_n": 14, "batch": 33, "ntt_form": True},
        # ciphertext x ciphertext of the serving mix
        {"name": "ct_mul_12x16384", "op": "ct_mul", "q": "q224", "log_n": 14, "batch": 12},
        # examples/fma.cpp at the size the benchmark reports
        {"name": "fma_2^24", "op": "fma", "q": "fma", "elements": 1 << 24},
        # hundreds of polynomials of uneven degree in one planned, captured launch
        {"name": "uneven_512", "op": "uneven", "q": "q192", "count": 512, "log_min": 12, "log_max": 16},
        # 4 x 4 matrices of NTT-form polynomials times vectors of them (linear layers on ciphertexts)
        {"name": "matvec_16x4x4", "op": "matvec", "q": "q256", "log_n": 15, "batch": 16, "rows": 4, "cols": 4},
        # the sum of a share vector of no particular length
        {"name": "sum_9999991", "op": "sum", "q": "fma", "elements": 9999991},
        # a tensor through the stream cipher, as it is before it leaves the machine
        {"name": "cipher_1000003", "op": "cipher", "q": "q160", "elements": 1000003},
        # a burst of mixed requests through the serving loop
        {"name": "serving_48", "op": "serving", "count": 48, "log_min": 12, "log_max": 14, "moduli": "q128,q256"},
    ]


def _log_uniform(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    op = rng.choice(["ntt", "keygen", "enc", "dec", "ct_mul", "fma", "uneven", "matvec", "sum", "cipher"])
    q = rng.choice(CIPHERTEXT_MODULI)
    log_n = rng.randint(12, 16)
    n = 1 << log_n
    if op == "ntt":
        return {"op": op, "q": rng.choice(["ntt"] + CIPHERTEXT_MODULI), "log_n": log_n,
                "batch": _log_uniform(rng, 1, (1 << 21) / n)}
    if op == "keygen":
        return {"op": op, "q": q, "log_n": log_n}
    if op == "enc":
        return {"op": op, "q": q, "log_n": log_n, "batch": _log_uniform(rng, 1, (1 << 21) / n),
                "tuned": rng.random() < 0.5, "ntt_form": rng.random() < 0.5}
    if op in ("dec", "ct_mul"):
        c = {"op": op, "q": q, "log_n": log_n, "batch": _log_uniform(rng, 1, (1 << 21) / n)}
        if op == "dec":
            c["ntt_form"] = rng.random() < 0.5
        return c
    if op == "uneven":
        return {"op": op, "q": q, "count": _log_uniform(rng, 16, 300), "log_min": 12, "log_max": rng.randint(13, 16)}
    if op == "matvec":
        rows, cols = rng.randint(1, 6), rng.randint(1, 6)
        return {"op": op, "q": q, "log_n": log_n, "batch": _log_uniform(rng, 1, (1 << 21) / n / 6), "rows": rows,
                "cols": cols}
    return {"op": op, "q": rng.choice(["fma"] + CIPHERTEXT_MODULI), "elements": _log_uniform(rng, 1000, 1 << 24)}


def _words(generator, limbs, elements, top):
    """limb-planar residues: uniform limbs, the top one below the modulus's own"""
    x = torch.randint(-(1 << 31), 1 << 31, (limbs, elements), dtype=torch.int64, device="cuda", generator=generator)
    x[-1] = torch.randint(0, top, (elements,), dtype=torch.int64, device="cuda", generator=generator)
    return torch.where(x >= 1 << 31, x - (1 << 32), x).to(torch.int32)


class _State:
    """what a program keeps: its queue, moduli and inputs"""

    def __init__(self, seed):
        rng = random.Random(seed)
        self.queue = Queue(key=[rng.getrandbits(32) for _ in range(8)])
        self.nonce = [rng.getrandbits(32), rng.getrandbits(32), 1]
        self.rng = rng
        self.generator = torch.Generator(device="cuda")
        self.generator.manual_seed(seed)

    def residues(self, modulus, shape, n=1):
        t = Tensor(modulus, shape, n, torch.empty((modulus.limbs, int(np.prod(shape, dtype=np.int64)) * n),
                                                  dtype=torch.int32, device="cuda"))
        t.data.copy_(_words(self.generator, modulus.limbs, t.elements, modulus.value >> (32 * (modulus.limbs - 1))))
        return t


def _uneven_degrees(case):
    rng = random.Random(case["count"])
    return [1 << rng.randint(case["log_min"], case["log_max"]) for _ in range(case["count"])]


def prepare(case, seed):
    s = _State(seed)
    s.case, op, queue = case, case["op"], s.queue
    if op == "serving":
        return _prepare_serving(s)
    q = s.q = queue.modulus(MODULI[case["q"]])
    if op in ("fma", "sum", "cipher"):
        s.x = s.residues(q, (case["elements"],))
        if op == "fma":
            s.y, s.z = s.residues(q, (case["elements"],)), s.residues(q, (case["elements"],))
            s.out = Tensor(q, (case["elements"],))
        elif op == "cipher":
            s.key, s.stream_nonce = queue.key[::-1], s.nonce
        return s
    if op == "uneven":
        # the same degrees for every seed, so that a batch is the same work; the data differs
        s.degrees = _uneven_degrees(case)
        whole = s.residues(q, (sum(s.degrees),)).data
        s.inputs, s.outputs, at = [], [], 0
        out = torch.empty(q.limbs * sum(s.degrees), dtype=torch.int32, device="cuda")
        for n in s.degrees:
            s.inputs.append(Tensor(q, (), n, whole[:, at:at + n].contiguous()))
            s.outputs.append(Tensor(q, (), n, out[q.limbs * at:q.limbs * (at + n)].view(q.limbs, n)))
            at += n
        s.out = out
        s.plan = NttBatch(queue, q, s.degrees)
        return s
    n = 1 << case["log_n"]
    batch = case.get("batch", 1)
    if op == "ct_mul":
        s.x = lhe.Ciphertext(s.residues(q, (batch,), n), s.residues(q, (batch,), n))
        s.y = lhe.Ciphertext(s.residues(q, (batch,), n), s.residues(q, (batch,), n))
        return s
    if op == "matvec":
        s.m = s.residues(q, (batch, case["rows"], case["cols"]), n)
        s.x = s.residues(q, (batch, case["cols"]), n)
        s.out = Tensor(q, (batch, case["rows"]), n)
        return s
    q.prepare(n)
    if op == "ntt":
        q.tune(n, batch)
        q.tune(n, batch, inverse=True)
        s.x, s.y, s.z = s.residues(q, (batch,), n), Tensor(q, (batch,), n), Tensor(q, (batch,), n)
        return s
    p = s.p = queue.modulus(P)
    p.prepare(n)
    if op == "keygen":
        q.tune(n, 1)
    elif op == "enc":
        if case["tuned"]:
            q.tune(n, batch)
            p.tune(n, batch, inverse=True)
        s.key = lhe.Key(s.residues(q, (), n), s.residues(q, (), n))
        s.x = s.residues(p, (batch,), n)
        s.out = lhe.Ciphertext(Tensor(q, (batch,), n), Tensor(q, (batch,), n))
    elif op == "dec":
        q.tune(n, batch, inverse=True)
        if case["ntt_form"]:
            p.tune(n, batch)
        s.secret = queue.ntt_centered_binomial(q, n, (), 1)
        s.x = lhe.Ciphertext(s.residues(q, (batch,), n), s.residues(q, (batch,), n))
        s.out = Tensor(p, (batch,), n)
    return s


def _serving_requests(case, seed):
    return serving.poisson_stream(case["count"], seed=seed, log_n=(case["log_min"], case["log_max"]),
                                  moduli=case["moduli"].split(","))


def _prepare_serving(s):
    case, queue = s.case, s.queue
    # the same shapes for every seed, so that a burst is the same work; the data differs.  Every
    # request's results are slices of one buffer
    arrivals = _serving_requests(case, 1)
    p = queue.modulus(P)
    keys = {}
    s.server = serving.Server(queue, memory_budget=1 << 30)
    results = {serving.REQUEST_NTT: 1, serving.REQUEST_ENCRYPT: 2, serving.REQUEST_CT_MUL: 3}
    words = [LIMBS[a.q] * a.count << a.log_n for a in arrivals for _ in range(results[a.kind])]
    s.out = torch.empty(sum(words), dtype=torch.int32, device="cuda")
    slices = iter(torch.split(s.out, words))
    s.requests = []
    for a in arrivals:
        n = 1 << a.log_n
        q = queue.modulus(MODULI[a.q])
        q.prepare(n)
        p.prepare(n)
        outs = [Tensor(q, (a.count,), n, next(slices).view(q.limbs, a.count * n)) for _ in range(results[a.kind])]
        if a.kind == serving.REQUEST_NTT:
            s.requests.append((s.server.submit_ntt, (q, s.residues(q, (a.count,), n), *outs)))
        elif a.kind == serving.REQUEST_ENCRYPT:
            if (a.q, n) not in keys:
                key = lhe.Key(s.residues(q, (), n), s.residues(q, (), n))
                keys[a.q, n] = (key, s.server.add_key(q, p, key))
            x = s.residues(p, (a.count,), n)
            s.requests.append((s.server.submit_encrypt, (keys[a.q, n][1], q, x, *outs, [a.index, s.nonce[0], 1])))
        else:
            operands = [s.residues(q, (a.count,), n) for _ in range(4)]
            s.requests.append((s.server.submit_ct_mul, (q, *operands, *outs)))
    s.keys = keys
    queue.wait()
    return s


def run(s):
    op, queue = s.case["op"], s.queue
    if op == "ntt":
        queue.ntt(s.x, out=s.y)
        queue.intt(s.y, out=s.z)
        return [s.y.data, s.z.data]
    if op == "keygen":
        queue.nonce = s.nonce
        secret, key = lhe.keygen(queue, s.q, s.p, 1 << s.case["log_n"])
        return [secret.data, key.a.data, key.b.data]
    if op == "enc":
        queue.nonce = s.nonce
        lhe.enc(queue, s.key, s.x, s.q, plaintext_ntt=s.case["ntt_form"], out=s.out)
        return [s.out.c0.data, s.out.c1.data]
    if op == "dec":
        return lhe.dec(queue, s.secret, s.x, s.p, plaintext_ntt=s.case["ntt_form"], out=s.out).data
    if op == "ct_mul":
        z = lhe.mul(queue, s.x, s.y)
        return [z.c0.data, z.c1.data, z.c2.data]
    if op == "fma":
        return queue.fma(s.x, s.y, s.z, out=s.out).data
    if op == "uneven":
        s.plan.run(s.inputs, s.outputs)
        return s.out
    if op == "matvec":
        return queue.matrix_vector_product(s.m, s.x, out=s.out).data
    if op == "sum":
        return queue.sum(s.x).data
    if op == "cipher":
        return queue.cipher_enc(s.key, s.stream_nonce, s.x)
    for submit, arguments in s.requests:
        submit(*arguments)
    s.server.drain()
    return s.out


def exact(case, seed):
    """Every result is a tensor of whole words, the one right answer bit for bit: there is no error to measure."""
    return None


def work(case):
    """bytes: every operand and result once; flops: two for each 32-bit multiply of the exact products"""
    op = case["op"]
    if op == "serving":
        total = {"bytes": 0.0, "flops": 0.0}
        kinds = {serving.REQUEST_NTT: "half", serving.REQUEST_ENCRYPT: "enc", serving.REQUEST_CT_MUL: "ct_mul"}
        for a in _serving_requests(case, 1):
            w = work({"op": kinds[a.kind], "q": a.q, "log_n": a.log_n, "batch": a.count, "ntt_form": False})
            total = {k: total[k] + w[k] for k in total}
        return total
    limbs = LIMBS[case["q"]]
    product = 2.0 * (4 * limbs * limbs + limbs)  # one Montgomery product
    p_limbs = LIMBS["p64"]
    p_product = 2.0 * (4 * p_limbs * p_limbs + p_limbs)
    if op in ("fma", "sum", "cipher"):
        e = case["elements"]
        return {"bytes": 4.0 * limbs * e * {"fma": 4, "sum": 1, "cipher": 2}[op],
                "flops": product * e if op == "fma" else 0.0}
    if op == "uneven":
        degrees = _uneven_degrees(case)
        return {"bytes": 8.0 * limbs * sum(degrees),
                "flops": product * sum(n / 2 * (n.bit_length() - 1) for n in degrees)}
    n = 1 << case["log_n"]
    e = n * case.get("batch", 1)
    transform = case["log_n"] / 2  # products per element
    if op in ("ntt", "half"):
        times = 2 if op == "ntt" else 1
        return {"bytes": times * 8.0 * limbs * e, "flops": times * product * transform * e}
    if op == "keygen":
        return {"bytes": 4.0 * limbs * 3 * e, "flops": product * (2 * transform + 2) * e}
    if op == "enc":
        return {"bytes": 4.0 * (2 * limbs * (e + n) + p_limbs * e),
                "flops": (product * (3 * transform + 2) + (p_product * transform if case["ntt_form"] else 0)) * e}
    if op == "dec":
        return {"bytes": 4.0 * (limbs * (2 * e + n) + p_limbs * e),
                "flops": (product * (transform + 1) + (p_product * transform if case["ntt_form"] else 0)) * e}
    if op == "ct_mul":
        return {"bytes": 4.0 * limbs * 7 * e, "flops": product * 4 * e}
    cells = e * case["rows"] * case["cols"]
    return {"bytes": 4.0 * limbs * (cells + e * (case["rows"] + case["cols"])), "flops": product * cells}
