"""The multiplications a user of this library runs, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program holds before the call (operands
and the context, batch or server it keeps), `run` is one pass through the Python binding of the
C ABI.  Kinds of call:
  device  Multiplier.multiply_device: `count` products of operands already in device memory
  static  Multiplier.multiply_device_static: one product, nothing allocated
  host    Multiplier.multiply: one product of host operands over PCIe (page-locked with pinned)
  batch   Batch.run: classes of uneven points, one CUDA-graph launch
  server  Server.run: requests from pinned host memory against operands resident on the device
Coefficients are below q, L = ceil(W / 32) little-endian 32-bit limbs each.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polymult-challenge_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import polymult  # noqa: E402
import workload  # noqa: E402


def listed():
    return [
        # one small product: launches and latency are all there is
        {"name": "device 4096/256 x1", "kind": "device", "N": 4096, "W": 256, "count": 1, "values": "uniform"},
        # many small products in one call
        {"name": "device 4096/256 x64", "kind": "device", "N": 4096, "W": 256, "count": 64, "values": "uniform"},
        # a ragged point: W one above a multiple of 8, an odd count of products
        {"name": "device 8192/1001 x5", "kind": "device", "N": 8192, "W": 1001, "count": 5, "values": "uniform"},
        # the middle point, one product at a time (a program that depends on each result) and batched
        {"name": "device 32768/868 x1", "kind": "device", "N": 32768, "W": 868, "count": 1, "values": "uniform"},
        {"name": "device 32768/868 x16", "kind": "device", "N": 32768, "W": 868, "count": 16, "values": "uniform"},
        # the ranked point, one product and a full launch group
        {"name": "device 65536/1747 x1", "kind": "device", "N": 65536, "W": 1747, "count": 1, "values": "uniform"},
        {"name": "device 65536/1747 x32", "kind": "device", "N": 65536, "W": 1747, "count": 32, "values": "uniform"},
        # a wide modulus (more primes than one tensor-core tile holds)
        {"name": "device 65536/3000 x4", "kind": "device", "N": 65536, "W": 3000, "count": 4, "values": "uniform"},
        # the reference's call: one product of pageable host vectors
        {"name": "host 65536/1747", "kind": "host", "N": 65536, "W": 1747, "pinned": False, "values": "uniform"},
        # one product of page-locked host operands, 1% of the coefficients nonzero
        {"name": "host pinned 32768/868", "kind": "host", "N": 32768, "W": 868, "pinned": True, "values": "sparse"},
        # multiplications of uneven points in one graph launch
        {"name": "batch uneven", "kind": "batch", "points": "4096/256x12 8192/868x8 16384/256x6 16384/1747x4 "
         "4096/3000x5 32768/868x4 65536/1747x2 16384/3000x2", "values": "uniform"},
        # a burst of requests against resident operands
        {"name": "server 16384/1747 x24", "kind": "server", "N": 16384, "W": 1747, "count": 24, "resident": 4,
         "values": "uniform"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# residue words (coefficients x primes) of a drawn case at most: half the largest listed case's, since
# a word costs up to twice as much at the widest moduli
_MOST_WORDS = 16 * 118 * 65536


def draw(rng):
    """N a power of two in [2048, 65536], W any width in [64, 4000], one to 64 products."""
    def point(most=_MOST_WORDS):
        while True:
            N, W = 1 << rng.randint(11, 16), _log_int(rng, 64, 4000)
            if N * _primes(N, W) <= most:
                return N, W

    kind = rng.choice(["device"] * 6 + ["static", "host", "host", "batch", "server"])
    values = rng.choice(["uniform", "uniform", "uniform", "sparse", "small", "largest"])
    if kind == "batch":
        pts = []
        for _ in range(rng.randint(2, 6)):
            N, W = point()
            pts.append("%d/%dx%d" % (N, W, _log_int(rng, 1, max(1, min(16, _MOST_WORDS // 6 // (N * _primes(N, W)))))))
        return {"kind": kind, "points": " ".join(pts), "values": values}
    # the static call's fixed scratch holds 8 Mi residue words per operand
    N, W = point(8 << 20 if kind == "static" else _MOST_WORDS)
    if kind == "static":
        return {"kind": kind, "N": N, "W": W, "count": 1, "values": values}
    if kind == "host":
        return {"kind": kind, "N": N, "W": W, "pinned": rng.random() < 0.5, "values": values}
    count = _log_int(rng, 1, max(1, min(64, _MOST_WORDS // (N * _primes(N, W)))))
    if kind == "server":
        count = max(2, min(count, 32, (64 << 20) // (N * _limbs(W) * 4)))
        return {"kind": kind, "N": N, "W": W, "count": count, "resident": rng.randint(1, 8), "values": values}
    return {"kind": kind, "N": N, "W": W, "count": count, "values": values}


def _limbs(W):
    return (W + 31) // 32


def _primes(N, W):
    """RNS primes below 2^30 that an exact product needs: their product passes 8 N q^2."""
    return -(-(2 * W + N.bit_length() + 2) // 30)


def _modulus(N, W):
    """The spec-derived prime where the library lists it, else the largest number below 2^W that
    is 1 mod 2N: the library takes any odd modulus just below 2^W, and its primality changes nothing."""
    if (N, W) in workload.SPEC_DELTAS:
        return workload.spec_prime(N, W)
    return (1 << W) - 2 * N + 1


def _points(case):
    """[(N, W, count)] of a case."""
    if case["kind"] == "batch":
        out = []
        for p in case["points"].split():
            nw, c = p.split("x")
            N, W = nw.split("/")
            out.append((int(N), int(W), int(c)))
        return out
    return [(case["N"], case["W"], case.get("count", 1))]


def _operands(N, W, count, values, seed):
    """[count, N, L] int32 tensor of limbs on the GPU, every coefficient in [0, q): a uniform
    W-bit value is below q but for a share of at most 2^-40 of the draws."""
    L, q = _limbs(W), _modulus(N, W)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if values == "largest":  # every coefficient q - 1, the first of each operand drawn
        x = torch.from_numpy(workload.limbs(q - 1, L).view(np.int32)).cuda().repeat(count, N, 1)
        x[:, 0] = _operands(1, W, count, "uniform", seed)[:, 0]
        return x
    if values == "small":  # below 2^16
        x = torch.zeros(count, N, L, dtype=torch.int32, device="cuda")
        x[:, :, 0] = torch.randint(0, 1 << 16, (count, N), dtype=torch.int32, device="cuda", generator=g)
        return x
    x = torch.randint(-(1 << 31), 1 << 31, (count, N, L), dtype=torch.int32, device="cuda", generator=g)
    if W % 32:
        x[:, :, -1] &= (1 << (W % 32)) - 1
    if values == "sparse":  # 1% of the coefficients nonzero
        keep = torch.rand(count, N, 1, device="cuda", generator=g) < 0.01
        keep[:, 0] = True
        x *= keep
    return x


def _pair(N, W, count, values, seed):
    return (_operands(N, W, count, values, 2 * seed + 1_000_003), _operands(N, W, count, values, 2 * seed + 1_000_004))


def prepare(case, seed):
    kind, values = case["kind"], case["values"]
    state = {"kind": kind}
    if kind == "batch":
        state["ops"], classes = [], []
        for i, (N, W, count) in enumerate(_points(case)):
            a, b = _pair(N, W, count, values, seed + 7919 * i)
            c = torch.zeros_like(a)
            state["ops"].append((a, b, c))
            classes.append((N, W, workload.limbs(_modulus(N, W), _limbs(W)), count, a.data_ptr(), b.data_ptr(),
                            c.data_ptr()))
        state["batch"] = polymult.Batch(classes)
        return state
    N, W, count = _points(case)[0]
    L = _limbs(W)
    q = workload.limbs(_modulus(N, W), L)
    if kind == "server":
        a, _ = _pair(N, W, count, values, seed)
        res = _operands(N, W, case["resident"], values, 3 * seed + 17).cpu().numpy().view(np.uint32)
        state["server"] = polymult.Server(N, W, q, res)
        # page-locked buffers of the program's own, which outlive the server
        state["a"] = a.cpu().pin_memory().numpy().view(np.uint32)
        state["c"] = torch.zeros(a.shape, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        state["t"] = np.zeros(count)
        state["sel"] = np.random.default_rng(seed).integers(0, case["resident"], size=count).astype(np.uint32)
        return state
    a, b = _pair(N, W, count, values, seed)
    state["m"], state["count"] = polymult.Multiplier(N, W, q), count
    if kind == "host":
        def host(x):
            t = x[0].cpu()
            return (t.pin_memory() if case["pinned"] else t).numpy().view(np.uint32)
        state["a"], state["b"] = host(a), host(b)
        state["c"] = host(torch.zeros_like(a))
    else:
        state["a"], state["b"], state["c"] = a, b, torch.zeros_like(a)
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run(torch.cuda.current_stream().cuda_stream)
        return [c for _, _, c in state["ops"]]
    if kind == "server":
        state["server"].run(state["t"], state["sel"], list(state["a"]), list(state["c"]))
        return state["c"].view(np.int32)
    m, a, b, c = state["m"], state["a"], state["b"], state["c"]
    if kind == "host":
        return m.multiply(a, b, out=c).view(np.int32)
    s = torch.cuda.current_stream().cuda_stream
    if kind == "static":
        m.multiply_device_static(a.data_ptr(), b.data_ptr(), c.data_ptr(), s)
    else:
        m.multiply_device(a.data_ptr(), b.data_ptr(), c.data_ptr(), state["count"], s)
    return c


def work(case):
    """Bytes: operands in, products out.  Operations: the 32-bit multiplies and adds of a product
    over K primes -- the transforms' butterflies (3 multiplies, 3 adds each), the pointwise products
    and the decompositions' and the CRT's limb-by-prime multiply-adds; a resident operand's
    decomposition and transform are not part of a request."""
    n_in, n_tr = (1, 2) if case["kind"] == "server" else (2, 3)
    total_b = total_f = 0.0
    for N, W, count in _points(case):
        K, L, logN = _primes(N, W), _limbs(W), N.bit_length() - 1
        total_b += count * (n_in + 1) * 4.0 * N * L
        total_f += count * (n_tr * K * (N / 2) * logN * 6 + 6.0 * K * N + (n_in + 1) * 2.0 * K * N * L)
    return {"bytes": total_b, "flops": total_f}


def exact(case, seed):
    """Products of the smallest single products as one big integer multiplication each."""
    if case["kind"] not in ("device", "static", "host"):
        return None
    N, W, count = _points(case)[0]
    if count * (N * (2 * W + 20) / 2e6) ** 1.6 > 20:  # big-integer multiplication, seconds
        return None
    L, q = _limbs(W), _modulus(N, W)
    slot = (2 * W + N.bit_length() + 9) // 8  # bytes of one coefficient of the full product
    out = np.zeros((count, N, L), dtype=np.uint32)
    a, b = (x.cpu().numpy().view(np.uint8).reshape(count, N, 4 * L) for x in _pair(N, W, count, case["values"], seed))

    def joined(x):
        wide = np.zeros((N, slot), dtype=np.uint8)
        wide[:, :min(slot, 4 * L)] = x[:, :min(slot, 4 * L)]
        return int.from_bytes(wide.tobytes(), "little")

    for i in range(count):
        prod = (joined(a[i]) * joined(b[i])).to_bytes(2 * N * slot, "little")
        co = [int.from_bytes(prod[k * slot:(k + 1) * slot], "little") for k in range(2 * N)]
        for k in range(N):
            out[i, k] = workload.limbs((co[k] - co[k + N]) % q, L)
    out = out.view(np.int32)
    return out[0] if case["kind"] == "host" else out
