"""Performance cases of the IPFE library: the calls its users make, over the sizes they make them at.

Every case goes through the public Python API (cufe_b200.Context, Ring, Batch, SvmModel) on
device tensors, as a program that keeps its keys and ciphertexts on the GPU does.  `listed()`
are the fixed cases, `draw(rng)` gives others of the same kinds and ranges:

  encrypt   Context.encrypt / encrypt_gpu_map: 1..64 vectors under one master key
  setup     Context.setup / setup_gpu_map: one master key pair
  keygen    Context.keygen: 1..600 function keys from one master key
  decrypt   Context.decrypt + decode: some ciphertexts under some function keys
  svm       SvmModel.predict: test vectors against the support vectors' function keys
  ntt       Ring.forward and Ring.inverse over a stack of RNS polynomials
  batch     Batch.replay: one step over instances of uneven n and l

Outputs are whole numbers (residues, decoded inner products, labels), so they are compared
bit for bit; only the SVM's decision values are floating point, and `exact` computes those.
"""
import math

import numpy as np
import torch

import cufe_b200 as cf

DEV = "cuda:0"


def listed():
    return [
        # One short vector at the smallest ring in use: a call whose time is latency and launches.
        {"name": "encrypt_small", "kind": "encrypt", "mapping": "cpu", "n": 1024, "l": 32, "batch": 1},
        # One vector of 784 features (an MNIST image) per call: the plain per-call form.
        {"name": "encrypt_call", "kind": "encrypt", "mapping": "cpu", "n": 4096, "l": 784, "batch": 1},
        # The same vectors 40 at a time: the throughput form.
        {"name": "encrypt_batch", "kind": "encrypt", "mapping": "cpu", "n": 4096, "l": 784, "batch": 40},
        # The device part of the drop-in rlwe_sife_encrypt_gpu at its default length: some test
        # vectors in one call, one seed for all.
        {"name": "encrypt_gpu_map", "kind": "encrypt", "mapping": "gpu", "n": 4096, "l": 785, "batch": 8},
        # A master key pair at the default length (the reference's timing loop makes one per vector).
        {"name": "setup", "kind": "setup", "mapping": "cpu", "n": 4096, "l": 785},
        # One function key for signed weights: what a client asks for between two models.
        {"name": "keygen_one", "kind": "keygen", "n": 4096, "l": 784, "keys": 1, "signed": True},
        # The function keys of a model of 591 support vectors (the shipped a1a model's count).
        {"name": "keygen_model", "kind": "keygen", "n": 4096, "l": 785, "keys": 591, "signed": False},
        # A batch of ciphertexts under one key, every coefficient decoded.
        {"name": "decrypt_batch", "kind": "decrypt", "n": 4096, "l": 784, "cts": 40, "keys": 1, "signed": True, "coeffs": 4096},
        # One test vector against every support vector's key, as svm_predict_gpu calls it: the
        # full decryption, then coefficient 0 decoded.
        {"name": "decrypt_model", "kind": "decrypt", "n": 2048, "l": 124, "cts": 1, "keys": 591, "signed": False, "coeffs": 1},
        # 1,000 encrypted test vectors against 500 resident support vectors, with the vote.
        {"name": "svm_predict", "kind": "svm", "n": 2048, "l": 124, "cts": 1000, "classes": 2, "svs": 500},
        # A stack of RNS polynomials transformed in each direction.
        {"name": "ntt", "kind": "ntt", "n": 4096, "k": 3, "polys": 8192},
        # One graph replay of a mixed batch: encrypt, keygen and decrypt per instance, l from 32
        # to 1,024, n 2048 or 4096.
        {"name": "batch_mixed", "kind": "batch", "count": 96, "l_min": 32, "l_max": 1024},
    ]


def _log(rng, lo, hi):
    """a whole number in [lo, hi], uniform over its logarithm"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["encrypt", "encrypt", "encrypt", "setup", "keygen", "keygen", "decrypt", "decrypt", "svm", "ntt",
                       "ntt", "batch"])
    n = rng.choice([1024, 2048, 4096])
    l = _log(rng, 32, 1024)
    if kind == "encrypt":
        most = max(1, min(64, 40 * 784 * 4096 // (l * n)))
        return {"kind": kind, "mapping": rng.choice(["cpu", "cpu", "gpu"]), "n": n, "l": l, "batch": _log(rng, 1, most)}
    if kind == "setup":
        return {"kind": kind, "mapping": rng.choice(["cpu", "gpu"]), "n": n, "l": l}
    if kind == "keygen":
        return {"kind": kind, "n": n, "l": l, "keys": _log(rng, 1, 600), "signed": rng.random() < 0.5}
    if kind == "decrypt":
        l = _log(rng, 32, 800)
        cts = _log(rng, 1, max(1, min(64, 40 * 784 * 4096 // (l * n))))
        keys = _log(rng, 1, max(1, min(600, 40 * 784 * 4096 // (l * n * cts))))
        return {"kind": kind, "n": n, "l": l, "cts": cts, "keys": keys, "signed": rng.random() < 0.5,
                "coeffs": rng.choice([1, n])}
    if kind == "svm":
        return {"kind": kind, "n": rng.choice([1024, 2048]), "l": _log(rng, 32, 124), "cts": _log(rng, 16, 1000),
                "classes": rng.choice([2, 2, 3]), "svs": _log(rng, 16, 500)}
    if kind == "ntt":
        n, k = rng.choice([1024, 2048, 4096, 8192]), rng.randint(3, 6)
        return {"kind": kind, "n": n, "k": k, "polys": _log(rng, 1, 3 * 8192 * 4096 // (n * k))}
    return {"kind": kind, "count": _log(rng, 8, 96), "l_min": 32, "l_max": _log(rng, 128, 1024)}


# ------------------------------------------------------------------ inputs


def _seeds(rs, count):
    return rs.randint(0, 256, (count, 32)).astype(np.uint8)


def _a1a_rows(rs, cts, l):
    """binary test vectors with about 14 ones at 1-based features, as the a1a rows are"""
    x = np.zeros((cts, l), np.uint32)
    for t in range(cts):
        x[t, 1 + rs.choice(l - 1, min(14, l - 1), replace=False)] = 1
    return x


def _weights(rs, shape, signed):
    """quantised weights: signed in [-16, 16], or unsigned up to the scheme's bound 16"""
    return rs.randint(-16 if signed else 0, 17, shape).astype(np.int32)


def _svm_plain(case, seed):
    """the SVM case's plain data: test vectors, support vectors and the model"""
    rs = np.random.RandomState(seed % (1 << 31))
    svs, nr = case["svs"], case["classes"]
    nsv = [svs // nr + (1 if i < svs % nr else 0) for i in range(nr)]
    sv = _weights(rs, (svs, case["l"]), True)
    sv[:, 0] = 0
    x = _a1a_rows(rs, case["cts"], case["l"])
    coef = rs.uniform(-1, 1, (nr - 1, svs))
    rho = rs.uniform(-0.5, 0.5, nr * (nr - 1) // 2)
    return rs, x, sv, nsv, coef, rho, np.arange(nr, dtype=np.int32) * 2 - 1


def prepare(case, seed):
    kind = case["kind"]
    rs = np.random.RandomState(seed % (1 << 31))
    st = {"kind": kind, "case": case}
    if kind == "ntt":
        ring = cf.Ring(case["n"], case["k"])
        gen = torch.Generator(device=DEV).manual_seed(seed)
        q = torch.tensor(ring.primes.astype(np.int64), device=DEV).reshape(1, -1, 1)

        def residues():
            u = torch.randint(0, 2 ** 31 - 1, (case["polys"], case["k"], case["n"]), device=DEV, dtype=torch.int32,
                              generator=gen)
            return torch.remainder(u, q.to(torch.int32))

        st.update(ring=ring, coeffs=residues(), values=residues())
        return st
    if kind == "batch":
        cnt = case["count"]
        # the shapes are the case's own; only the data depends on the seed
        shape = np.random.RandomState(cnt + case["l_max"])
        l = np.rint(np.exp(shape.uniform(math.log(case["l_min"]), math.log(case["l_max"]), cnt))).astype(np.int32)
        n = np.where(shape.permutation(cnt) % 2 == 0, 2048, 4096).astype(np.int32)
        b = cf.Batch(n, l)
        b.setup(_seeds(rs, cnt), _seeds(rs, cnt), _seeds(rs, cnt))
        x = cf.to_dev(rs.randint(0, 5, int(l.sum())).astype(np.uint32))
        y = torch.from_numpy(_weights(rs, int(l.sum()), True)).to(DEV)
        d0 = torch.empty((cnt, 3), dtype=torch.int32, device=DEV)
        out = b.bind(x, y, cf.bytes_to_dev(_seeds(rs, cnt)), cf.bytes_to_dev(_seeds(rs, cnt)), d0=d0)
        st.update(batch=b, out=out, d0=d0)
        return st
    ctx = cf.Context(case["n"], case["l"])
    st["ctx"] = ctx
    if kind == "setup":
        st["seeds"] = _seeds(rs, 3)
        st["mpk"], st["msk"] = ctx.mpk_buf(), ctx.msk_buf()
        if case["mapping"] == "gpu":  # the caller's uniform polynomial a
            st["a"] = ctx.sample_polya(st["seeds"][0])
        return st
    if kind == "svm":
        rs, x, sv, nsv, coef, rho, label = _svm_plain(case, seed)
        mpk, msk = ctx.setup(*_seeds(rs, 3))
        st["model"] = cf.SvmModel(ctx, sv, nsv, coef, rho, label, msk)
        st["ct"] = ctx.encrypt(cf.to_dev(x), mpk, _seeds(rs, case["cts"]), _seeds(rs, case["cts"]))
        st["kvalue"] = torch.empty((case["cts"], case["svs"]), dtype=torch.int32, device=DEV)
        st["dec"] = torch.empty((case["cts"], len(rho)), dtype=torch.float64, device=DEV)
        return st
    mpk, msk = ctx.setup(*_seeds(rs, 3))
    if kind == "encrypt":
        b = case["batch"]
        st["x"] = cf.to_dev(rs.randint(0, 5, (b, case["l"])).astype(np.uint32))
        st["mpk"], st["ct"] = mpk, ctx.ct_buf(b)
        st["seeds2"], st["seeds3"] = _seeds(rs, b), _seeds(rs, b)
        return st
    st["y"] = torch.from_numpy(_weights(rs, (case["keys"], case["l"]), case["signed"])).to(DEV)
    if kind == "keygen":
        st["msk"] = msk
        return st
    cts = case["cts"]
    x = cf.to_dev(rs.randint(0, 5, (cts, case["l"])).astype(np.uint32))
    st["ct"] = ctx.encrypt(x, mpk, _seeds(rs, cts), _seeds(rs, cts))
    st["sky"] = ctx.keygen(st["y"], msk, y_signed=case["signed"])
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "ntt":
        return st["ring"].forward(st["coeffs"]), st["ring"].inverse(st["values"])
    if kind == "batch":
        st["batch"].replay()
        return st["out"], st["d0"]
    ctx = st["ctx"]
    if kind == "setup":
        if case["mapping"] == "gpu":
            return ctx.setup_gpu_map(st["a"], st["seeds"][1], st["seeds"][2], mpk=st["mpk"], msk=st["msk"])
        return ctx.setup(*st["seeds"], mpk=st["mpk"], msk=st["msk"])
    if kind == "svm":
        return {"label": st["model"].predict(st["ct"], kvalue=st["kvalue"], dec=st["dec"]), "kvalue": st["kvalue"],
                "dec": st["dec"]}
    if kind == "encrypt":
        if case["mapping"] == "gpu":
            return ctx.encrypt_gpu_map(st["x"], st["mpk"], st["seeds2"][0], ct=st["ct"])
        return ctx.encrypt(st["x"], st["mpk"], st["seeds2"], st["seeds3"], ct=st["ct"])
    if kind == "keygen":
        return ctx.keygen(st["y"], st["msk"], y_signed=case["signed"])
    dy = ctx.decrypt(st["ct"], st["y"], st["sky"], y_signed=case["signed"])
    return dy, ctx.decode(dy, ncoeff=case["coeffs"])


# ------------------------------------------------------------------ the work that a pass cannot do without


def _ntt_ops(n):
    """operations of one transform: log2(n) / 2 butterflies per coefficient, each a modular
    product, a sum and a difference"""
    return 1.5 * n * math.log2(n)


def work(case):
    """Bytes: each input read once, each output written once.  Operations: modular products and
    sums; the random bits of the samplers are not counted."""
    kind = case["kind"]
    if kind == "ntt":
        r = case["polys"] * case["k"]
        return {"bytes": 2 * 8 * r * case["n"], "flops": 2 * r * _ntt_ops(case["n"])}
    if kind == "batch":
        # mean l of the log-uniform lengths; per instance: mpk and msk read
        lm = (case["l_max"] - case["l_min"]) / math.log(case["l_max"] / case["l_min"])
        res = 3 * lm * case["count"]
        return {"bytes": 2 * 4 * res * 3072, "flops": res * (_ntt_ops(3072) + 6 * 3072)}
    n, l = case["n"], case["l"]
    poly = 3 * n
    if kind == "setup":
        return {"bytes": 4 * poly * (2 * l + 1), "flops": 3 * (2 * l + 1) * _ntt_ops(n) + 2 * l * poly}
    if kind == "encrypt":
        b = case["batch"]
        return {"bytes": 4 * (poly * (l + 1) * (1 + b) + b * l), "flops": b * 3 * (l + 2) * _ntt_ops(n) + b * 4 * l * poly}
    if kind == "keygen":
        k = case["keys"]
        return {"bytes": 4 * (poly * (l + k) + k * l), "flops": 2 * k * l * poly}
    if kind == "svm":
        c, k = case["cts"], case["svs"]
        # coefficient 0 of c_0 .. c_{l-1}, all of c_l; the function keys; kvalue and decisions
        return {"bytes": 4 * 3 * (c + k) * (l + n) + 4 * c * k, "flops": 2 * 3 * c * k * (l + n)}
    c, k = case["cts"], case["keys"]
    return {"bytes": 4 * (poly * (c * (l + 1) + k + c * k) + k * l + c * k * case["coeffs"]),
            "flops": 2 * c * k * l * poly + 3 * (2 * c * k + c + k) * _ntt_ops(n)}


def exact(case, seed):
    """The SVM's decision values from the plain vectors (every other output is a whole number)."""
    if case["kind"] != "svm":
        return None
    _, x, sv, nsv, coef, rho, _ = _svm_plain(case, seed)
    kv = (x.astype(np.int64) @ sv.T.astype(np.int64)).astype(np.float64)
    start = np.concatenate([[0], np.cumsum(nsv)])
    dec = []
    for i in range(len(nsv)):
        for j in range(i + 1, len(nsv)):
            a, b = slice(start[i], start[i + 1]), slice(start[j], start[j + 1])
            dec.append(kv[:, a] @ coef[j - 1][a] + kv[:, b] @ coef[i][b] - rho[len(dec)])
    return {"label": None, "kvalue": None, "dec": np.stack(dec, axis=1)}
