"""Timing cases of the encrypted Hamming kNN paths, through the public entry points.

Each case is a dict of plain values; ``prepare`` builds what a program holds
before the call (keys and tables installed on the device, the encrypted index,
the request), ``run`` makes one pass, ``exact`` gives the values that follow
from the plaintexts alone and ``work`` counts what a pass cannot do without.

Kinds and what they stand for:

* ``knn``      Paillier-Lookup search: encrypt the query batch, multiply it
               with every index ciphertext (encode_hamming_server), decode
               every distance.  Arrays on the device, as a server holds them.
* ``decode``   the client's decode of received products alone.
* ``index``    Paillier-Lookup encryption of an index (fixed-base tables).
* ``encrypt``, ``decrypt``  textbook Paillier over a batch.
* ``search``   BFV packed search of one encrypted query over an index kept on
               the device (``resident``) or passed as host bytes.
* ``client``   BFV client encryption of packed vectors to the wire format.

Keys are fixed per size (a program has one key for many calls); the inputs
come from the seed.
"""

from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from cuhepy_b200.bfv import _bfv_rns
from cuhepy_b200.bfv import layout as bfv_layout
from cuhepy_b200.paillier.gpu import NOISE_MULTIPLES, PaillierDevice

ALPHA = 280          # bits of the secret exponent of a lookup key
T = 65537            # BFV plaintext modulus
GADGET = 30          # BFV key-switch digit bits
TARGET_BITS = 50     # response modulus of a compacted search


def listed() -> list[dict]:
    return [
        # the smallest call: one client compares one pair of vectors
        {"name": "decode_one", "kind": "decode", "key_len": 1024, "embed": 512, "vectors": 1},
        # one interactive query against a small index, a size that fills no tile evenly
        {"name": "knn_small", "kind": "knn", "key_len": 1024, "embed": 512, "queries": 1, "vectors": 1003},
        # a batch of queries against a larger index: 65,536 distances
        {"name": "knn_batch", "kind": "knn", "key_len": 1024, "embed": 512, "queries": 4, "vectors": 16384},
        # bulk encryption of an index
        {"name": "index_bulk", "kind": "index", "key_len": 1024, "embed": 512, "vectors": 65536},
        # textbook Paillier: 4,096 values of 32 bits, encrypted and decrypted
        {"name": "encrypt_1024", "kind": "encrypt", "key_len": 1024, "count": 4096, "plain_bits": 32},
        {"name": "decrypt_1024", "kind": "decrypt", "key_len": 1024, "count": 4096, "plain_bits": 32},
        # the widest key, a short ragged batch; the narrowest key, a long one
        {"name": "encrypt_2048", "kind": "encrypt", "key_len": 2048, "count": 333, "plain_bits": 4000},
        {"name": "decrypt_512", "kind": "decrypt", "key_len": 512, "count": 20011, "plain_bits": 1000},
        # one query over 16,384 packed vectors kept on the device
        {"name": "search_resident", "kind": "search", "n": 8192, "q_bits": 180, "native": False, "embed": 512,
         "tiles": 1024, "resident": True, "compact": True},
        # the default client's ring (a prime modulus), a small index
        {"name": "search_native", "kind": "search", "n": 8192, "q_bits": 180, "native": True, "embed": 512,
         "tiles": 100, "resident": True, "compact": True},
        # the reference's own call form: the index as host bytes, a small ring, full responses
        {"name": "search_host", "kind": "search", "n": 4096, "q_bits": 120, "native": False, "embed": 256,
         "tiles": 37, "resident": False, "compact": False},
        # a client encrypts 500 vectors for the index
        {"name": "client_encrypt", "kind": "client", "n": 8192, "q_bits": 180, "embed": 512, "vectors": 500},
    ]


def _log(rng: random.Random, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["knn", "decode", "index", "encrypt", "decrypt", "search", "search", "client"])
    if kind in ("knn", "decode", "index"):
        case = {"kind": kind, "key_len": rng.choice([512, 1024, 1024]),
                "embed": rng.choice([96, 256, 384, 512, 768, 1024])}
        if kind == "knn":
            case["queries"] = _log(rng, 1, 16)
            case["vectors"] = _log(rng, 1, 65536 // case["queries"])
        else:
            case["vectors"] = _log(rng, 1, 65536)
        return case
    if kind in ("encrypt", "decrypt"):
        key_len = rng.choice([512, 1024, 2048])
        most = {512: 20000, 1024: 4096, 2048: 333}[key_len]
        return {"kind": kind, "key_len": key_len, "count": _log(rng, 1, most),
                "plain_bits": rng.choice([1, 32, key_len, 2 * key_len - 50])}
    if kind == "search":
        n, q_bits = rng.choice([(4096, 120), (8192, 180), (8192, 180), (16384, 300)])
        most = {4096: 1024, 8192: 1000, 16384: 160}[n]
        return {"kind": kind, "n": n, "q_bits": q_bits, "native": rng.random() < 0.3,
                "embed": rng.choice([100, 128, 256, 512, 1024]), "tiles": _log(rng, 1, most),
                "resident": rng.random() < 0.7, "compact": rng.random() < 0.7}
    n, q_bits = rng.choice([(4096, 120), (8192, 180), (16384, 300)])
    embed = rng.choice([128, 256, 512])
    return {"kind": kind, "n": n, "q_bits": q_bits, "embed": embed,
            "vectors": _log(rng, 1, 32 * bfv_layout.Layout(n, embed).capacity)}


# ---- Paillier keys (fixed per size) -----------------------------------------------
_SIEVE = [p for p in range(3, 5000, 2) if all(p % d for d in range(3, int(p ** 0.5) + 1, 2))]


def _is_prime(x: int) -> bool:
    if any(x % p == 0 for p in _SIEVE):
        return x in _SIEVE
    d, r = x - 1, 0
    while not d & 1:
        d, r = d >> 1, r + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19):
        y = pow(a, d, x)
        if y in (1, x - 1):
            continue
        for _ in range(r - 1):
            y = y * y % x
            if y == x - 1:
                break
        else:
            return False
    return True


def _prime(rng: random.Random, bits: int) -> int:
    while True:
        x = rng.getrandbits(bits) | 1 | (3 << (bits - 2))
        if _is_prime(x):
            return x


@functools.lru_cache(maxsize=None)
def _textbook_key(key_len: int) -> dict:
    rng = random.Random(1000 + key_len)
    p, q = _prime(rng, key_len), _prime(rng, key_len)
    n, phi = p * q, (p - 1) * (q - 1)
    return {"n": n, "p": p, "q": q, "exponent": phi, "multiplier": pow(phi, -1, n)}


@functools.lru_cache(maxsize=None)
def _lookup_key(key_len: int) -> dict:
    """An alpha-subgroup key: p = k q1 + 1, g of order a n, a = q1 q2."""
    rng = random.Random(2000 + key_len)

    def side(order_bits: int):
        order = _prime(rng, order_bits)
        low, high = (3 << (key_len - 2)) // order, (1 << key_len) // order
        while True:
            k = 2 * rng.randrange(low // 2, high // 2)
            p = k * order + 1
            if p.bit_length() == key_len and _is_prime(p):
                break
        while True:
            g = pow(rng.randrange(2, p - 1), (p - 1) // order, p)
            if g != 1:
                return p, order, g * (1 + p) % (p * p)

    p, q1, gp = side(ALPHA // 2)
    q, q2, gq = side(ALPHA - ALPHA // 2)
    n, a = p * q, q1 * q2
    n2 = n * n
    g = (gp + p * p * ((gq - gp) * pow(p * p, -1, q * q) % (q * q))) % n2
    noise, z, g_n = [], 1, pow(g, n, n2)
    for _ in range(256):
        z = z * z * g_n % n2
        noise.append(z)
    inverse = pow((pow(g, a, n2) - 1) // n, -1, n)
    return {"n": n, "p": p, "q": q, "exponent": a, "multiplier": inverse, "g": g, "noise": noise}


def _handle(key: dict) -> PaillierDevice:
    ctx = PaillierDevice(key["n"])
    ctx.set_secret(key["exponent"], key["multiplier"])
    ctx.set_factors(key["p"], key["q"])
    return ctx


@functools.lru_cache(maxsize=None)
def _textbook(key_len: int) -> PaillierDevice:
    return _handle(_textbook_key(key_len))


@functools.lru_cache(maxsize=None)
def _lookup(key_len: int) -> PaillierDevice:
    key = _lookup_key(key_len)
    ctx = _handle(key)
    ctx.build_tables(key["g"], key_len * 2 // 8, key["noise"])
    return ctx


def _chunks(case: dict) -> tuple[int, int]:
    chunk_len = 2 * case["key_len"]
    return chunk_len, max(1, -(-2 * case["embed"] // chunk_len))


def _cuda(array: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(array.view(np.int32) if array.dtype == np.uint32 else array).cuda()


def _bits(case: dict, seed: int, what: int, count: int) -> np.ndarray:
    return np.random.default_rng([seed, what]).integers(0, 2, size=(count, case["embed"]), dtype=np.uint8)


def _encrypt_inputs(case: dict, seed: int, what: int, count: int) -> dict:
    chunks = _chunks(case)[1]
    noise = np.random.default_rng([seed, what, 1]).integers(0, 256, size=(count * chunks, NOISE_MULTIPLES),
                                                            dtype=np.uint8)
    words = 4 * case["key_len"] // 32
    return {"bits": _cuda(_bits(case, seed, what, count)), "noise": _cuda(noise), "count": count,
            "out": torch.zeros((count * chunks, words), dtype=torch.int32, device="cuda")}


def _lookup_encrypt(ctx: PaillierDevice, case: dict, item: dict) -> torch.Tensor:
    chunk_len, chunks = _chunks(case)
    ctx.lookup_encrypt_bits_array(item["bits"], item["count"], case["embed"], chunk_len, chunks, item["noise"],
                                  item["out"])
    return item["out"]


def _integers(rng: np.random.Generator, count: int, bits: int, words: int) -> np.ndarray:
    """[count, words] limbs of integers of at most `bits` bits."""
    raw = rng.integers(0, 1 << 32, size=(count, words), dtype=np.uint32)
    full, rest = divmod(bits, 32)
    if full < words:
        raw[:, full] &= np.uint32((1 << rest) - 1)
        raw[:, full + 1:] = 0
    return raw


# ---- BFV handles ----------------------------------------------------------------------
def _modulus(case: dict) -> int:
    if case.get("native"):
        return bfv_layout.coefficient_modulus(case["q_bits"])
    return bfv_layout.rns_modulus(case["n"], case["q_bits"])


def _uniform_poly(rng: np.random.Generator, n: int, q: int) -> bytes:
    """n fixed-width coefficients below q (the top byte below q's)."""
    width = (q.bit_length() + 7) // 8
    raw = rng.integers(0, 256, size=(n, width), dtype=np.uint8)
    raw[:, -1] = rng.integers(0, q >> (8 * (width - 1)), size=n, dtype=np.uint8)
    return raw.tobytes()


def _packed(rng: np.random.Generator, n: int, bits: int) -> bytes:
    """n coefficients of bits - 1 random bits, packed `bits` bits each."""
    keep = np.ones((n, bits), dtype=np.uint8)
    keep[:, -1] = 0
    mask = np.packbits(keep.reshape(-1), bitorder="little")
    return (np.frombuffer(rng.bytes(mask.size), dtype=np.uint8) & mask).tobytes()


@functools.lru_cache(maxsize=None)
def _ring(n: int, q: int, native: bool):
    return _bfv_rns.create_ring(n, format(q, "x"), GADGET, True, not native, 0 if native else 2)


@functools.lru_cache(maxsize=4)
def _server(n: int, q: int, native: bool, embed: int):
    """A search server with uniform keys (the evaluation does not depend on their values)."""
    rng = np.random.default_rng([n, embed, native])
    layout = bfv_layout.Layout(n, embed)
    ring = _ring(n, q, native)
    digits = -(-q.bit_length() // GADGET)

    def key():
        return _bfv_rns.compile_key(ring, tuple((_uniform_poly(rng, n, q), _uniform_poly(rng, n, q))
                                                for _ in range(digits)))

    relin = key()
    galois = tuple((g, key()) for g in sorted(set(layout.left()) | set(layout.right())))
    target = format(bfv_layout.coefficient_modulus(TARGET_BITS), "x")
    return _bfv_rns.create_server(relin, galois, layout.padded, T, target), layout


# ---- states ---------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind in ("knn", "decode", "index"):
        ctx = _lookup(case["key_len"])
        chunks = _chunks(case)[1]
        vectors = case["vectors"]
        state = {"case": case, "ctx": ctx, "index": _encrypt_inputs(case, seed, 1, vectors)}
        if kind == "index":
            return state
        queries = case.get("queries", 1)
        state["query"] = _encrypt_inputs(case, seed, 2, queries)
        _lookup_encrypt(ctx, case, state["index"])
        _lookup_encrypt(ctx, case, state["query"])
        words = state["index"]["out"].shape[1]
        # chunk-major index rows: the products of a query's chunk c are those
        # with the index's chunks c, gathered into [query, vector, chunk]
        state["products"] = torch.zeros((queries * vectors * chunks, words), dtype=torch.int32, device="cuda")
        state["distances"] = torch.zeros(queries * vectors, dtype=torch.int64, device="cuda")
        ctx.synchronize()
        state["by_chunk"] = [state["index"]["out"].view(vectors, chunks, words)[:, c].contiguous()
                             for c in range(chunks)]
        torch.cuda.synchronize()
        _multiply(state)
        ctx.synchronize()
        return state
    if kind in ("encrypt", "decrypt"):
        ctx, count, words = _textbook(case["key_len"]), case["count"], 4 * case["key_len"] // 32
        rng = np.random.default_rng(seed)
        plain = _integers(rng, count, case["plain_bits"], words)
        # r below 2^(bits(n) - 1) <= n; a common factor with n has negligible probability
        r = _integers(rng, count, 2 * case["key_len"] - 1, words)
        r[:, 0] |= 1
        state = {"case": case, "ctx": ctx, "count": count, "m": _cuda(plain), "r": _cuda(r),
                 "out": torch.zeros((count, words), dtype=torch.int32, device="cuda")}
        if kind == "decrypt":
            state["c"] = torch.zeros_like(state["out"])
            torch.cuda.synchronize()
            ctx.encrypt_array(state["m"], state["r"], state["c"], count)
            ctx.synchronize()
        return state
    n, q = case["n"], _modulus(case)
    rng = np.random.default_rng(seed)
    if kind == "search":
        server, layout = _server(n, q, case["native"], case["embed"])
        bits = q.bit_length()
        index = tuple((_packed(rng, n, bits), _packed(rng, n, bits)) for _ in range(case["tiles"]))
        # the last tile is part full unless a tile holds two vectors only
        vectors = case["tiles"] * layout.capacity - seed % max(1, layout.capacity // 2)
        state = {"case": case, "server": server, "vectors": vectors, "query": (_packed(rng, n, bits), _packed(rng, n, bits))}
        state["index"] = _bfv_rns.upload_index(server, index) if case["resident"] else index
        return state
    layout = bfv_layout.Layout(n, case["embed"])
    ring = _ring(n, q, False)
    slots = layout.index_slots(rng.integers(0, 2, size=(case["vectors"], case["embed"]), dtype=np.uint8))
    return {"case": case, "ring": ring, "slots": slots, "key": rng.bytes(32), "nonce": rng.bytes(12),
            "public": (_uniform_poly(rng, n, q), _uniform_poly(rng, n, q))}


def _multiply(state: dict) -> None:
    """encode_hamming_server of every query with every index vector, chunk by chunk."""
    ctx, query, vectors = state["ctx"], state["query"], state["case"]["vectors"]
    chunks = len(state["by_chunk"])
    if chunks == 1:
        ctx.mulmod_outer_array(query["out"], query["count"], state["by_chunk"][0], vectors, state["products"])
        return
    words = query["out"].shape[1]
    parts = []
    for c in range(chunks):
        q = query["out"].view(-1, chunks, words)[:, c].contiguous()
        part = torch.empty((query["count"] * vectors, words), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ctx.mulmod_outer_array(q, query["count"], state["by_chunk"][c], vectors, part)
        parts.append(part)
    state["products"].copy_(torch.stack(parts, 1).view_as(state["products"]))
    torch.cuda.synchronize()


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind in ("knn", "decode", "index"):
        ctx = state["ctx"]
        if kind == "index":
            return _lookup_encrypt(ctx, case, state["index"])
        chunk_len, chunks = _chunks(case)
        if kind == "knn":
            _lookup_encrypt(ctx, case, state["query"])
            if chunks > 1:
                ctx.synchronize()  # the chunks are gathered by torch, on its own stream
            _multiply(state)
        ctx.decode_array(state["products"], state["distances"].numel(), chunks, chunk_len, state["distances"])
        if kind == "decode":
            return state["distances"]
        return {"query": state["query"]["out"], "products": state["products"], "distances": state["distances"]}
    if kind == "encrypt":
        state["ctx"].encrypt_array(state["m"], state["r"], state["out"], state["count"])
        return state["out"]
    if kind == "decrypt":
        state["ctx"].decrypt_array(state["c"], state["out"], state["count"])
        return state["out"]
    if kind == "search":
        search = _bfv_rns.search_index if case["resident"] else _bfv_rns.packed_search
        if case["resident"]:
            responses = search(state["server"], state["index"], state["query"], state["vectors"], case["compact"])
        else:
            responses = search(state["server"], state["query"], state["index"], state["vectors"], case["compact"])
        return [np.frombuffer(part, dtype=np.uint8) for pair in responses for part in pair]
    wire = _bfv_rns.encrypt_packed_keyed(state["ring"], state["public"], T, state["slots"], state["key"],
                                         state["nonce"])
    return [np.frombuffer(part, dtype=np.uint8) for pair in wire for part in pair]


# ---- exact values ---------------------------------------------------------------------
def _limbs(values: list[int], words: int) -> torch.Tensor:
    raw = b"".join(v.to_bytes(4 * words, "little") for v in values)
    return torch.from_numpy(np.frombuffer(raw, dtype=np.int32).reshape(len(values), words).copy())


def _lookup_ciphertexts(case: dict, seed: int, what: int, count: int) -> torch.Tensor | None:
    """g^m times the drawn noise entries, for as many ciphertexts as Python does in seconds."""
    chunk_len, chunks = _chunks(case)
    if count * chunks > 128:
        return None
    key = _lookup_key(case["key_len"])
    n2 = key["n"] ** 2
    noise = np.random.default_rng([seed, what, 1]).integers(0, 256, size=(count * chunks, NOISE_MULTIPLES),
                                                            dtype=np.uint8)
    out = []
    for v, row in enumerate(_bits(case, seed, what, count)):
        text = "".join("0" + str(int(b)) for b in row)
        for c in range(chunks):
            x = pow(key["g"], int(text[c * chunk_len:(c + 1) * chunk_len], 2), n2)
            for k in noise[v * chunks + c]:
                x = x * key["noise"][int(k)] % n2
            out.append(x)
    return _limbs(out, 4 * case["key_len"] // 32)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "index":
        return _lookup_ciphertexts(case, seed, 1, case["vectors"])
    if kind in ("knn", "decode"):
        queries = case.get("queries", 1)
        index, query = _bits(case, seed, 1, case["vectors"]), _bits(case, seed, 2, queries)
        distances = torch.from_numpy(np.stack([(index ^ q).sum(1, dtype=np.int64) for q in query]).reshape(-1))
        if kind == "decode":
            return distances
        return {"query": _lookup_ciphertexts(case, seed, 2, queries), "products": None, "distances": distances}
    if kind in ("encrypt", "decrypt"):
        words, count = 4 * case["key_len"] // 32, case["count"]
        rng = np.random.default_rng(seed)
        plain = _integers(rng, count, case["plain_bits"], words)
        if kind == "decrypt":
            return torch.from_numpy(plain.view(np.int32))
        if count * case["key_len"] ** 3 > 16 * 2048 ** 3:
            return None
        r = _integers(rng, count, 2 * case["key_len"] - 1, words)
        r[:, 0] |= 1
        n = _textbook_key(case["key_len"])["n"]
        n2 = n * n
        values = [(1 + int.from_bytes(a.tobytes(), "little") * n) * pow(int.from_bytes(b.tobytes(), "little"), n, n2)
                  % n2 for a, b in zip(plain, r)]
        return _limbs(values, words)
    return None  # ciphertext bytes: no value but the circuit's own


# ---- work -----------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Bytes in and out; operations as 32-bit multiply-adds (two each) of the
    products mod n^2, or of the transforms' butterflies."""
    kind = case["kind"]
    if kind in ("search", "client"):
        n, primes = case["n"], case["q_bits"] // 60
        packed = n * case["q_bits"] // 8
        butterfly = n / 2 * math.log2(n) * 10 * 2
        layout = bfv_layout.Layout(n, case["embed"])
        if kind == "client":
            cts = -(-case["vectors"] // layout.capacity)
            return {"bytes": cts * (4 * n + 2 * packed), "flops": cts * (1 + 3 * primes) * butterfly}
        digits = -(-case["q_bits"] // GADGET)
        switches = case["tiles"] * (1 + len(layout.left())) + case["tiles"]
        response = n * (TARGET_BITS if case["compact"] else case["q_bits"]) // 8
        groups = -(-case["tiles"] // layout.padded)
        keys = (1 + 2 * len(layout.left())) * digits * 2 * primes * n * 8
        return {"bytes": (case["tiles"] + 1) * 2 * packed + 2 * groups * response + keys,
                "flops": (switches * (digits + 1) * primes + case["tiles"] * 5 * (2 * primes + 1)) * butterfly}
    words = 4 * case["key_len"] // 32
    product = 2 * 2 * words * words      # one modular product, multiply and reduce
    if kind in ("encrypt", "decrypt"):
        steps = 2 * case["key_len"] * 1.15
        # decryption knows the factors: two half-width powers of half the exponent's length
        per = steps * product if kind == "encrypt" else 2 * (steps / 2) * product / 4
        return {"bytes": case["count"] * words * 4 * (3 if kind == "encrypt" else 2), "flops": case["count"] * per}
    chunks = _chunks(case)[1]
    table = (min(case["embed"], case["key_len"]) / 8 + NOISE_MULTIPLES) * product
    decode = ALPHA * 1.2 * 2 * product / 4
    vectors = case["vectors"]
    if kind == "index":
        return {"bytes": vectors * (case["embed"] + chunks * (NOISE_MULTIPLES + 4 * words)),
                "flops": vectors * chunks * table}
    pairs = case.get("queries", 1) * vectors
    if kind == "decode":
        return {"bytes": pairs * (chunks * 4 * words + 8), "flops": pairs * chunks * decode}
    queries = case["queries"]
    return {"bytes": (vectors + queries + pairs) * chunks * 4 * words + pairs * 8,
            "flops": queries * chunks * table + pairs * chunks * (product + decode)}
