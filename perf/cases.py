"""The work that programs have this library do, as cases that can be timed and compared.

A case names an entry point (`op`), its data type, a ring size 2^n_power and a
batch. `listed()` has the ones that stand for real use, `draw(rng)` gives more of
the same ranges: rings 2^10 (drop-in: 2^12, its smallest) .. 2^20, batches from
one product to a few hundred megabytes of operands, odd ones among them.

`prepare` makes what a program holds before the call (operands, twiddle tables,
workspace, plan); `run` is one pass through the public entry points; `work` is
what a pass cannot do without; `exact` is the same result from torch's 64-bit
transforms.
"""
import importlib.util
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory ``gpu-fft_b200/``, imported as ``gpufft_b200``."""
    if "gpufft_b200" not in sys.modules:
        d = os.path.join(ROOT, "gpu-fft_b200")
        spec = importlib.util.spec_from_file_location("gpufft_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gpufft_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["gpufft_b200"]


def listed():
    return [
        # One polynomial product per call through the reference's two calls, the
        # size of its own GPU example (test_ffnt_gpu_R_R: N = 2^12): latency.
        {"name": "ffnt_f64_2e12_b1", "op": "ffnt", "dtype": "f64", "n_power": 12, "batch": 1},
        # The same two calls as a homomorphic-encryption program batches them.
        {"name": "ffnt_f64_2e16_b256", "op": "ffnt", "dtype": "f64", "n_power": 16, "batch": 256},
        # Long complex transforms (C_C, forward both, inverse with the product) of
        # a signal-processing program, few of them; 2^20 is the middle of the
        # benchmark programs' upper axis.
        {"name": "fft_cc_f32_2e20_b11", "op": "fft_cc", "dtype": "f32", "n_power": 20, "batch": 11},
        # Zero-padded real polynomial products (R_R), double precision, ragged batch.
        {"name": "fft_rr_f64_2e14_b75", "op": "fft_rr", "dtype": "f64", "n_power": 14, "batch": 75},
        # The fused negacyclic product at the headline size, double precision.
        {"name": "negacyclic_f64_2e16_b256", "op": "negacyclic", "dtype": "f64", "n_power": 16, "batch": 256},
        # Small rings in large batches (bootstrapping-sized: 2^11), single precision.
        {"name": "negacyclic_f32_2e11_b4001", "op": "negacyclic", "dtype": "f32", "n_power": 11, "batch": 4001},
        # The exact integer product at the headline size: 24-bit coefficients.
        {"name": "split_2e16_b256_24bit", "op": "split", "dtype": "f32", "n_power": 16, "batch": 256, "bits": 24,
         "non_negative": True},
        # The exact product of a scheme with 16-bit signed digits in rings 2^13.
        {"name": "split_2e13_b333_16bit", "op": "split", "dtype": "f32", "n_power": 13, "batch": 333, "bits": 16,
         "non_negative": False},
        # Complex cyclic products of an ordinary batch, double precision.
        {"name": "cyclic_f64_2e14_b150", "op": "cyclic", "dtype": "f64", "n_power": 14, "batch": 150},
        # A long-convolution layer's training step: forward and both gradients.
        {"name": "conv_vjp_f32_2e14_b512", "op": "conv_vjp", "dtype": "f32", "n_power": 14, "batch": 512},
        # 4096 requests of mixed rings 2^10 .. 2^17 from a captured graph.
        {"name": "mixed_f64_4096", "op": "mixed", "dtype": "f64", "n_power": 17, "batch": 4096},
        # CKKS encoding and decoding (the canonical embedding) of 2^15 slots.
        {"name": "special_f64_2e15_b65", "op": "special", "dtype": "f64", "n_power": 15, "batch": 65},
    ]


# the most coefficients (points) per operand a drawn case of each kind has
_MOST = {"ffnt": 24, "fft_cc": 23, "fft_rr": 23, "negacyclic": 24, "split": 24, "cyclic": 23, "conv_vjp": 23,
         "special": 23}


def draw(rng):
    op = rng.choice(list(_MOST) + ["mixed"])
    c = {"op": op, "dtype": "f32" if op == "conv_vjp" else rng.choice(["f32", "f64", "f64"])}
    if op == "mixed":
        c["n_power"] = rng.randint(12, 17)
        c["batch"] = int(2 ** rng.uniform(4, 12))
        return c
    lo = 12 if op in ("ffnt", "fft_cc", "fft_rr") else 11 if op == "special" else 10
    hi = 17 if op == "split" and c["dtype"] == "f64" else 19 if op == "conv_vjp" else 20
    c["n_power"] = rng.randint(lo, hi)
    total = rng.uniform(c["n_power"], _MOST[op])  # log2 of the coefficients per operand
    c["batch"] = max(1, int(2 ** (total - c["n_power"])))
    if op == "split":
        c["bits"] = rng.randint(8, 24)
        c["non_negative"] = rng.random() < 0.5
    return c


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _real(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _cplx(case):
    return torch.complex128 if case["dtype"] == "f64" else torch.complex64


def _mixed_sizes(case):
    """log-uniform ring sizes 2^10 .. 2^n_power, the same for every seed (a server's request mix)."""
    r = random.Random(case["batch"] * 31 + case["n_power"])
    return [r.randint(10, case["n_power"]) for _ in range(case["batch"])]


def _coefficients(shape, bits, signed, dtype, g):
    lo, hi = (-(1 << (bits - 1)), 1 << (bits - 1)) if signed else (0, 1 << bits)
    return torch.randint(lo, hi, shape, dtype=torch.int32, device="cuda", generator=g).to(dtype)


def _operands(case, seed):
    """The call's inputs, from the seed alone."""
    g = _gen(seed)
    op, n, b = case["op"], 1 << case["n_power"], case["batch"]
    if op in ("ffnt", "negacyclic"):  # 16-bit coefficients, held as floating point (the reference's products)
        x = _coefficients((2 * b, n), 16, True, _real(case), g)
        return {"ab": x} if op == "ffnt" else {"a": x[:b], "b": x[b:]}
    if op == "fft_rr":  # the upper half of every row is the zero padding
        x = _coefficients((2 * b, n), 16, True, _real(case), g)
        x[:, n // 2:] = 0
        return {"ab": x}
    if op == "fft_cc":
        return {"ab": torch.randn(2 * b, n, dtype=_cplx(case), device="cuda", generator=g)}
    if op == "cyclic":
        x = torch.randn(2 * b, n, dtype=_cplx(case), device="cuda", generator=g)
        return {"a": x[:b], "b": x[b:]}
    if op == "special":  # slot values of a message
        return {"z": torch.randn(b, n, dtype=_cplx(case), device="cuda", generator=g)}
    if op == "split":
        x = _coefficients((2 * b, n), case["bits"], not case["non_negative"], torch.int32, g)
        return {"a": x[:b], "b": x[b:]}
    if op == "conv_vjp":
        x = torch.randn(4 * b, n, dtype=torch.float32, device="cuda", generator=g)
        return {"a": x[:b], "b": x[b:2 * b], "g": x[2 * b:].view(b, 2 * n)}
    total = sum(1 << k for k in _mixed_sizes(case))
    x = _coefficients((2, total), 16, True, _real(case), g)
    return {"a": x[0], "b": x[1]}


def _special_tables(n_power, dtype):
    """The canonical embedding's twiddles: entry t + j of span t is zeta^(5^j mod 8t), zeta = e^(2 pi i / 8t)."""
    tab = torch.zeros(1 << n_power, dtype=torch.complex128)
    for e in range(n_power):
        t = 1 << e
        p, q = 1, []
        for _ in range(t):
            q.append(p)
            p = p * 5 % (8 * t)
        ang = torch.tensor(q, dtype=torch.float64) * (2 * math.pi / (8 * t))
        tab[t:2 * t] = torch.polar(torch.ones_like(ang), ang)
    return tab.to(dtype), tab.conj().resolve_conj().to(dtype)


def prepare(case, seed):
    G = _package()
    op, n, b, k = case["op"], 1 << case["n_power"], case["batch"], case["n_power"]
    dt = case["dtype"]
    s = {"case": case, **_operands(case, seed)}
    cuda = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    if op == "ffnt":
        roots, inv_roots, twist, untwist = (cuda(t) for t in G.host_ffnt_tables(n, dt))
        s.update(roots=roots, inv_roots=inv_roots, twist=twist, untwist=untwist,
                 temp=torch.empty(2 * b * (n // 2), dtype=_cplx(case), device="cuda"), out=torch.empty_like(s["ab"][:b]))
        scale = 1.0 / (n // 2)
    elif op in ("fft_cc", "fft_rr"):
        roots, inv_roots, _ = G.host_fft_tables(n // 2, dt)
        s.update(roots=cuda(roots), inv_roots=cuda(inv_roots))
        if op == "fft_cc":
            s["buf"] = torch.empty_like(s["ab"])
        else:
            s["temp"] = torch.empty(2 * b * n, dtype=_cplx(case), device="cuda")
            s["out"] = torch.empty_like(s["ab"][:b])
        scale = 1.0 / n
    if op in ("ffnt", "fft_cc", "fft_rr"):
        s["fwd"] = G.fft_configuration(n_power=k, fft_type=G.FORWARD, reduction_poly=G.X_N_minus,
                                       zero_padding=op == "fft_rr")
        s["inv"] = G.fft_configuration(n_power=k, fft_type=G.INVERSE, reduction_poly=G.X_N_minus,
                                       mod_inverse=complex(scale))
        return s

    def workspace(nbytes):
        return torch.empty(nbytes, dtype=torch.uint8, device="cuda") if nbytes else None

    L, bits = G.lib(), 64 if dt == "f64" else 32
    if op == "negacyclic":
        s.update(tables=G.ffnt_tables(k, dt), out=torch.empty_like(s["a"]),
                 ws=workspace(G.negacyclic_mul_workspace_bytes(k, b, bits)))
    elif op == "cyclic":
        s.update(tables=G.ffnt_tables(k + 1, dt), out=torch.empty_like(s["a"]),
                 ws=workspace(int(L.gpufft_cyclic_mul_workspace_bytes(k, b, bits))))
    elif op == "split":
        limbs = G.split_plan(k, case["bits"], case["non_negative"], dt)
        need = (L.gpufft_negacyclic_mul_split_f64_workspace_bytes if dt == "f64" else
                L.gpufft_negacyclic_mul_split_workspace_bytes)(k, b, limbs[1])
        s.update(tables=G.ffnt_tables(k, dt), limbs=limbs, ws=workspace(int(need)),
                 out=torch.empty(b, n, dtype=torch.int64, device="cuda"))
    elif op == "conv_vjp":
        s.update(tables=G.ffnt_tables(k + 1, dt), out=torch.empty(b, 2 * n, dtype=torch.float32, device="cuda"),
                 ga=torch.empty_like(s["a"]), gb=torch.empty_like(s["b"]),
                 ws=workspace(max(int(L.gpufft_linear_mul_workspace_bytes(k, b, 32)),
                                  int(L.gpufft_linear_mul_vjp_workspace_bytes(k, b)))))
    elif op == "special":
        tab, inv_tab = _special_tables(k, _cplx(case))
        s.update(tab=tab.cuda(), inv_tab=inv_tab.cuda(), enc=torch.empty_like(s["z"]), dec=torch.empty_like(s["z"]),
                 fwd=G.fft_configuration(n_power=k, fft_type=G.FORWARD),
                 inv=G.fft_configuration(n_power=k, fft_type=G.INVERSE, mod_inverse=complex(1.0 / n)))
    elif op == "mixed":
        s["plan"] = G.BatchPlan(_mixed_sizes(case), _real(case))
        s["out"] = torch.empty_like(s["a"])
        s["plan"].autotune(s["a"], s["b"], s["out"])
        s["stream"] = torch.cuda.Stream()
        s["stream"].wait_stream(torch.cuda.current_stream())
        s["plan"].capture(s["a"], s["b"], s["out"], s["stream"])
    return s


def run(s):
    G = _package()
    op, b = s["case"]["op"], s["case"]["batch"]
    if op == "ffnt":
        G.GPU_FFNT(s["ab"], s["temp"], s["twist"], s["roots"], s["fwd"], 2 * b, False)
        G.GPU_FFNT(s["out"], s["temp"], s["untwist"], s["inv_roots"], s["inv"], b, True)
        return s["out"]
    if op == "fft_rr":
        G.GPU_FFT(s["ab"], s["temp"], s["roots"], s["fwd"], 2 * b, False)
        G.GPU_FFT(s["out"], s["temp"], s["inv_roots"], s["inv"], b, True)
        return s["out"]
    if op == "fft_cc":  # in place: the program keeps its operands
        s["buf"].copy_(s["ab"])
        G.GPU_FFT(s["buf"], s["roots"], s["fwd"], 2 * b, False)
        G.GPU_FFT(s["buf"], s["inv_roots"], s["inv"], b, True)
        return s["buf"][:b]
    if op == "negacyclic":
        return G.negacyclic_mul(s["a"], s["b"], out=s["out"], tables=s["tables"], workspace=s["ws"])
    if op == "cyclic":
        return G.cyclic_mul(s["a"], s["b"], out=s["out"], tables=s["tables"], workspace=s["ws"])
    if op == "split":
        c = s["case"]
        return G.negacyclic_mul_split(s["a"], s["b"], out=s["out"], input_bits=c["bits"],
                                      non_negative=c["non_negative"], limbs=s["limbs"], tables=s["tables"],
                                      workspace=s["ws"], precision=c["dtype"])
    if op == "conv_vjp":
        c = G.linear_mul(s["a"], s["b"], out=s["out"], tables=s["tables"], workspace=s["ws"])
        ga, gb = G.linear_mul_vjp(s["g"], s["a"], s["b"], grad_a=s["ga"], grad_b=s["gb"], tables=s["tables"],
                                  workspace=s["ws"])
        return {"c": c, "ga": ga, "gb": gb}
    if op == "special":  # encode into the ring, decode back
        s["enc"].copy_(s["z"])
        G.GPU_Special_FFT(s["enc"], s["inv_tab"], s["inv"], b)
        s["dec"].copy_(s["enc"])
        G.GPU_Special_FFT(s["dec"], s["tab"], s["fwd"], b)
        return {"enc": s["enc"], "dec": s["dec"]}
    s["plan"].replay(s["stream"])
    return s["out"]


def work(case):
    """Operands read once, results written once; 5 M log2 M per complex transform of M points and 6 per product."""
    op, n, b, k = case["op"], 1 << case["n_power"], case["batch"], case["n_power"]
    e = 8 if case["dtype"] == "f64" else 4

    def product(m, transforms=3):
        return transforms * 5 * (1 << m) * m + 6 * (1 << m)

    if op in ("ffnt", "negacyclic"):
        return {"bytes": 3 * b * n * e, "flops": b * product(k - 1)}
    if op == "fft_rr":  # half of each operand is padding
        return {"bytes": 2 * b * n * e, "flops": b * product(k - 1)}
    if op in ("fft_cc", "cyclic"):
        return {"bytes": 3 * b * n * 2 * e, "flops": b * product(k)}
    if op == "special":
        return {"bytes": 3 * b * n * 2 * e, "flops": b * 2 * 5 * n * k}
    if op == "split":
        return {"bytes": b * n * 16, "flops": b * product(k - 1)}
    if op == "conv_vjp":  # a, b, g in; c, grad_a, grad_b out
        return {"bytes": 8 * b * n * 4, "flops": b * 2 * product(k, 6)}
    sizes = _mixed_sizes(case)
    return {"bytes": 3 * e * sum(1 << j for j in sizes), "flops": sum(product(j - 1) for j in sizes)}


def _rows(f, *x):
    """f on a few rows at a time (64-bit spectra of a whole batch would not need to fit)."""
    step = max(1, (1 << 22) // x[0].shape[1])
    return torch.cat([f(*(y[i:i + step] for y in x)) for i in range(0, x[0].shape[0], step)])


def _linear(a, b):
    n = a.shape[1]
    return torch.fft.irfft(torch.fft.rfft(a.double(), 2 * n) * torch.fft.rfft(b.double(), 2 * n), 2 * n)


def _negacyclic(a, b):
    n = a.shape[1]
    w = torch.polar(torch.ones(n, dtype=torch.float64, device=a.device),
                    torch.arange(n, dtype=torch.float64, device=a.device) * (math.pi / n))
    return (torch.fft.ifft(torch.fft.fft(a.double() * w) * torch.fft.fft(b.double() * w)) * w.conj()).real.contiguous()


def _negacyclic_int(a, b):
    """Exact modulo 2^64: 12-bit digits, every digit product far below 2^53."""
    a, b = a.long(), b.long()
    a0, b0 = a & 4095, b & 4095
    a1, b1 = a >> 12, b >> 12
    lo, hi = (torch.round(_negacyclic(x, y)).long() for x, y in ((a0, b0), (a1, b1)))
    mid = torch.round(_negacyclic(a0, b1) + _negacyclic(a1, b0)).long()
    return lo + (mid << 12) + (hi << 24)


def _special(x, tab, inverse):
    n = x.shape[1]
    spans = [1 << e for e in range(n.bit_length() - 1)]
    for t in reversed(spans) if inverse else spans:
        v = x.view(x.shape[0], n // (2 * t), 2, t)
        w = tab[t:2 * t]
        u, l = (v[:, :, 0], v[:, :, 1]) if inverse else (v[:, :, 0], v[:, :, 1] * w)
        x = torch.stack((u + l, (u - l) * w if inverse else u - l), 2).reshape(x.shape[0], n)
    return x / n if inverse else x


def exact(case, seed):
    op, b, x = case["op"], case["batch"], _operands(case, seed)
    if op in ("ffnt", "fft_rr", "fft_cc"):
        p, q = x["ab"][:b], x["ab"][b:]
    if op == "ffnt":
        return _rows(_negacyclic, p, q)
    if op == "fft_rr":
        h = p.shape[1] // 2
        return _rows(_linear, p[:, :h], q[:, :h])
    if op in ("fft_cc", "cyclic"):
        p, q = (p, q) if op == "fft_cc" else (x["a"], x["b"])
        c128 = torch.complex128
        return _rows(lambda u, v: torch.fft.ifft(torch.fft.fft(u.to(c128)) * torch.fft.fft(v.to(c128))), p, q)
    if op == "negacyclic":
        return _rows(_negacyclic, x["a"], x["b"])
    if op == "split":
        return _rows(_negacyclic_int, x["a"], x["b"])
    if op == "conv_vjp":
        n = x["a"].shape[1]

        def grad(g, y):  # grad_a[i] = sum_k g[k] b[k - i]
            G, Y = torch.fft.rfft(g.double(), 4 * n), torch.fft.rfft(y.double(), 4 * n)
            return torch.fft.irfft(G * Y.conj(), 4 * n)[:, :n]

        return {"c": _rows(_linear, x["a"], x["b"]), "ga": _rows(grad, x["g"], x["b"]),
                "gb": _rows(grad, x["g"], x["a"])}
    if op == "special":
        tab, inv_tab = (t.cuda() for t in _special_tables(case["n_power"], torch.complex128))
        enc = _rows(lambda z: _special(z.to(torch.complex128), inv_tab, True), x["z"])
        return {"enc": enc, "dec": _rows(lambda z: _special(z, tab, False), enc)}
    # mixed: the packed operands are grouped by ring size, smallest first
    out, at, sizes = [], 0, _mixed_sizes(case)
    for k in sorted(set(sizes)):
        end = at + (sizes.count(k) << k)
        out.append(_rows(_negacyclic, x["a"][at:end].view(-1, 1 << k), x["b"][at:end].view(-1, 1 << k)).reshape(-1))
        at = end
    return torch.cat(out)
