"""The work that users of clpeak-b200 have it do, as cases whose speed can be compared between versions.

Three paths, each through the C ABI that the backend, the tests and the benchmark call:

* ``gemm``      one clpk_gemm of operands that are already on the device in the kernel's format: the GEMM rows;
* ``operands``  one matrix of operands made on the device: clpk_fill_f32, then clpk_convert_f32, or clpk_absmax_f32
                and clpk_quantize_fp4 for the block-scaled formats -- what stands in front of every GEMM row;
* ``stream``    one step of the bandwidth benchmark: read, copy and triad over three arrays, and the checksum read back.

A case is a dict: ``path``, and ``dtype`` / ``m`` / ``n`` / ``k`` / ``packed`` (gemm: the FP4 kinds' scales are already in
tile order), ``dtype`` / ``rows`` / ``cols`` (operands) or ``variant`` / ``floats`` (stream).
"""
import ctypes as C
import math

import numpy as np
import torch

from clpeak_b200 import native as N

DTYPES = {"bf16": N.DT_BF16, "f16": N.DT_F16, "e4m3": N.DT_E4M3, "e5m2": N.DT_E5M2, "tf32": N.DT_TF32, "i8": N.DT_I8,
          "nvf4": N.DT_NVF4, "mxf4": N.DT_MXF4, "f32": N.DT_F32, "f64": N.DT_F64}
VARIANTS = {"wide": N.STREAM_WIDE, "ldg": N.STREAM_LDG, "tma": N.STREAM_TMA}
BITS = {"bf16": 16, "f16": 16, "e4m3": 8, "e5m2": 8, "tf32": 32, "i8": 8, "nvf4": 4, "mxf4": 4, "f32": 32, "f64": 64}
OUT = {"tf32": torch.float32, "f32": torch.float32, "i8": torch.int32, "f64": torch.float64}     # bf16 for the others
SCALE_BLOCK = {"nvf4": 16, "mxf4": 32}
STREAM_BYTES = 1 << 33                # the benchmark's 8 GiB per array


def gemm(name, dtype, m, n, k, packed=False):
    return {"name": name, "path": "gemm", "dtype": dtype, "m": m, "n": n, "k": k, "packed": packed}


def listed():
    return [
        # the smallest call: the GEMM of the smoke test, where launch latency is the whole time
        gemm("gemm_bf16_512x256x512", "bf16", 512, 256, 512),
        # odd sizes that are no multiple of any tile, whole-number results
        gemm("gemm_i8_1000x1016x528", "i8", 1000, 1016, 528),
        # an ordinary small product, one wave of tiles or less
        gemm("gemm_e4m3_1024x1024x2048", "e4m3", 1024, 1024, 2048),
        # the smallest size of the GEMM configuration, in its first data type
        gemm("gemm_bf16_4096", "bf16", 4096, 4096, 4096),
        # the largest one, which is also the size the command line picks by itself
        gemm("gemm_e4m3_16384", "e4m3", 16384, 16384, 16384),
        # block-scaled operands that are new in every call: their scales arrive row-major and the call arranges them
        gemm("gemm_nvf4_2048", "nvf4", 2048, 2048, 2048),
        # block-scaled operands that stay: scales arranged once, as the backend's own row does
        gemm("gemm_nvf4_8192_packed", "nvf4", 8192, 8192, 8192, True),
        # the two rows without a tcgen05 kind
        gemm("gemm_f32_4096", "f32", 4096, 4096, 4096),
        gemm("gemm_f64_2048x2048x512", "f64", 2048, 2048, 512),
        # operands of one block-scaled GEMM of the configuration's middle size
        {"name": "operands_nvf4_8192", "path": "operands", "dtype": "nvf4", "rows": 8192, "cols": 8192},
        # operands of a small ragged GEMM
        {"name": "operands_e4m3_513x1040", "path": "operands", "dtype": "e4m3", "rows": 513, "cols": 1040},
        # the headline benchmark's step
        {"name": "stream_wide_8GiB", "path": "stream", "variant": "wide", "floats": STREAM_BYTES // 4},
    ]


def spread(rng, lo, hi, unit=1):
    """A multiple of `unit` in [lo, hi], even over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // unit, max(-(-lo // unit), round(v / unit))) * unit


def draw(rng):
    path = rng.choices(("gemm", "operands", "stream"), (8, 2, 2))[0]
    if path == "stream":
        return {"path": path, "variant": rng.choice(sorted(VARIANTS)), "floats": spread(rng, 1 << 14, STREAM_BYTES // 4, 4)}
    dtype = rng.choice(sorted(DTYPES))
    if path == "operands":
        unit = 64 if dtype in SCALE_BLOCK else 16
        return {"path": path, "dtype": dtype, "rows": spread(rng, 64, 16384), "cols": spread(rng, 128, 16384, unit)}
    # a row of A, of B and of C is a multiple of 16 bytes; the FP4 kinds take K in whole scale tiles
    k_unit = 256 if dtype in SCALE_BLOCK else 128 // BITS[dtype]
    n_unit = 1 if dtype in ("f32", "f64") else 4 if dtype in OUT else 8
    # no case above the largest listed one: the wide types have less arithmetic to offer
    most = {"f64": 2 ** 32, "f32": 2 ** 35, "tf32": 2 ** 40}.get(dtype, 2 ** 41)
    while True:
        m, n, k = spread(rng, 64, 16384), spread(rng, 64, 16384, n_unit), spread(rng, 256, 16384, k_unit)
        if m * n * k <= most:
            return {"path": path, "dtype": dtype, "m": m, "n": n, "k": k,
                    "packed": dtype in SCALE_BLOCK and rng.random() < 0.5}


def bytes_on_gpu(n):
    return torch.empty(max(int(n), 16), dtype=torch.uint8, device="cuda")


def operand(K, dtype, rows, cols, seed, stream):
    """(elements, scale bytes or None, tensor scale) of a rows x cols matrix from N(0, 0.02), int8 uniform in [-8, 7]."""
    if dtype == "i8":
        q = bytes_on_gpu(rows * cols)
        K.clpk_fill_i8(q.data_ptr(), rows * cols, seed, stream)
        return q, None, 1.0
    f = torch.empty(rows * cols, dtype=torch.float32, device="cuda")
    K.clpk_fill_f32(f.data_ptr(), rows * cols, seed, N.DIST_NORMAL, 0.0, 0.02, stream)
    if dtype == "f32":
        return f, None, 1.0
    q = bytes_on_gpu(rows * cols * BITS[dtype] // 8)
    if dtype not in SCALE_BLOCK:
        K.clpk_convert_f32(q.data_ptr(), f.data_ptr(), rows * cols, DTYPES[dtype], stream)
        return q, None, 1.0
    scale = 1.0
    if dtype == "nvf4":
        top = torch.empty(1, dtype=torch.float32, device="cuda")
        K.clpk_absmax_f32(top.data_ptr(), f.data_ptr(), rows * cols, stream)
        scale = float(np.float32(top.item()) / np.float32(6.0 * 448.0))
    sf = bytes_on_gpu(rows * cols // SCALE_BLOCK[dtype])
    K.clpk_quantize_fp4(q.data_ptr(), sf.data_ptr(), f.data_ptr(), rows, cols, DTYPES[dtype], scale, stream)
    return q, sf, scale


def prepare_gemm(K, case, seed, stream):
    dtype, m, n, k = case["dtype"], case["m"], case["n"], case["k"]
    a, sfa, scale_a = operand(K, dtype, m, k, 2 * seed, stream)
    b, sfb, scale_b = operand(K, "e4m3" if dtype == "e5m2" else dtype, n, k, 2 * seed + 1, stream)
    c = torch.empty(m, n, dtype=OUT.get(dtype, torch.bfloat16), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    need = C.c_size_t(0)
    K.clpk_gemm_workspace_bytes(DTYPES[dtype], m, n, k, C.byref(need))
    workspace = bytes_on_gpu(need.value)
    args = N.GemmArgs(dtype=DTYPES[dtype], m=m, n=n, k=k, d_a=a.data_ptr(), d_b=b.data_ptr(), d_c=c.data_ptr(),
                      d_sfa=sfa.data_ptr() if sfa is not None else None, d_sfb=sfb.data_ptr() if sfb is not None else None,
                      alpha=float(np.float32(scale_a) * np.float32(scale_b)), d_workspace=workspace.data_ptr(),
                      workspace_bytes=need.value, d_status=status.data_ptr())
    if case["packed"]:
        K.clpk_gemm_pack_scales(C.byref(args), stream)
        args.d_sfa = args.d_sfb = None
    return {"args": args, "c": c, "status": status, "keep": (a, b, sfa, sfb, workspace)}


def prepare_operands(case, seed):
    n, dtype = case["rows"] * case["cols"], case["dtype"]
    return {"rows": case["rows"], "cols": case["cols"], "dtype": dtype, "seed": seed,
            "f32": torch.empty(n, dtype=torch.float32, device="cuda"),
            "packed": bytes_on_gpu(n * BITS[dtype] // 8),
            "scales": bytes_on_gpu(n // SCALE_BLOCK[dtype]) if dtype in SCALE_BLOCK else None,
            "absmax": torch.empty(1, dtype=torch.float32, device="cuda")}


def prepare_stream(K, case, seed, stream):
    n = case["floats"]
    a, b, c, copied = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(4))
    for i, t in enumerate((b, c)):
        K.clpk_fill_f32(t.data_ptr(), n, 2 * seed + i, N.DIST_UNIFORM01, 0.0, 1.0, stream)
    grid = C.c_int(0)
    K.clpk_stream_read_grid(VARIANTS[case["variant"]], C.byref(grid))
    return {"variant": VARIANTS[case["variant"]], "n": n, "a": a, "b": b, "c": c, "copied": copied,
            "partials": torch.zeros(grid.value, dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    K = N.kernels()
    stream = torch.cuda.current_stream().cuda_stream
    if case["path"] == "gemm":
        state = prepare_gemm(K, case, seed, stream)
    elif case["path"] == "operands":
        state = prepare_operands(case, seed)
    else:
        state = prepare_stream(K, case, seed, stream)
    return dict(state, K=K, stream=stream, path=case["path"])


def run_operands(s):
    K, stream, n, dtype = s["K"], s["stream"], s["rows"] * s["cols"], s["dtype"]
    if dtype == "i8":
        K.clpk_fill_i8(s["packed"].data_ptr(), n, s["seed"], stream)
        return {"packed": s["packed"]}
    K.clpk_fill_f32(s["f32"].data_ptr(), n, s["seed"], N.DIST_NORMAL, 0.0, 0.02, stream)
    if dtype == "f32":
        return {"f32": s["f32"]}
    if dtype not in SCALE_BLOCK:
        K.clpk_convert_f32(s["packed"].data_ptr(), s["f32"].data_ptr(), n, DTYPES[dtype], stream)
        return {"f32": s["f32"], "packed": s["packed"]}
    scale = 1.0
    if dtype == "nvf4":               # the tensor scale is an argument, so the maximum comes to the host first
        K.clpk_absmax_f32(s["absmax"].data_ptr(), s["f32"].data_ptr(), n, stream)
        scale = float(np.float32(s["absmax"].item()) / np.float32(6.0 * 448.0))
    K.clpk_quantize_fp4(s["packed"].data_ptr(), s["scales"].data_ptr(), s["f32"].data_ptr(), s["rows"], s["cols"],
                        DTYPES[dtype], scale, stream)
    return {"f32": s["f32"], "packed": s["packed"], "scales": s["scales"], "tensor_scale": scale}


def run_stream(s):
    K, stream, v, n = s["K"], s["stream"], s["variant"], s["n"]
    K.clpk_stream_read(v, s["b"].data_ptr(), n * 4, s["partials"].data_ptr(), stream)
    K.clpk_stream_copy(v, s["copied"].data_ptr(), s["c"].data_ptr(), n * 4, stream)
    K.clpk_stream_triad(v, s["a"].data_ptr(), s["b"].data_ptr(), s["c"].data_ptr(), 1.5, n, stream)
    # which word of the partials holds what is the kernel's affair; their XOR is the checksum
    checksum = int(np.bitwise_xor.reduce(s["partials"].cpu().numpy()))
    return {"copied": s["copied"], "triad": s["a"], "checksum": checksum}


def run(state):
    if state["path"] == "gemm":
        state["K"].clpk_gemm(C.byref(state["args"]), state["stream"])
        return {"c": state["c"], "status": state["status"]}
    return run_operands(state) if state["path"] == "operands" else run_stream(state)


def work(case):
    if case["path"] == "stream":
        n = case["floats"]
        # read and copy's source once, triad's two operands, the two results
        return {"bytes": 6 * 4 * n, "flops": 2 * n}
    dtype = case["dtype"]
    scales = 1.0 / SCALE_BLOCK[dtype] if dtype in SCALE_BLOCK else 0.0
    per_element = BITS[dtype] / 8 + scales
    if case["path"] == "operands":
        n = case["rows"] * case["cols"]
        # the floats are a result too (written, and read once by the conversion); int8 and fp32 are made in place
        return {"bytes": n * (per_element if dtype in ("i8", "f32") else per_element + 8), "flops": 0}
    m, n, k = case["m"], case["n"], case["k"]
    out = OUT.get(dtype, torch.bfloat16).itemsize
    return {"bytes": (m + n) * k * per_element + m * n * out, "flops": 2 * m * n * k}


def tolerance(case):
    """Generated operands, copies and whole-number products are exact.  Floating products: about four times what one
    result shows against the same product in 64 bits -- for bf16 results that is the rounding of the result (2^-9
    at most; measured 1.7e-3 in the 2-norm), for tf32 and fp32 the sum over K (measured at K = 8192: 1.9e-5 and 1.6e-6),
    for fp64 the order of the sum."""
    if case["path"] != "gemm" or case["dtype"] == "i8":
        return "exact"
    if case["dtype"] == "f64":
        return {"rel": 1e-14, "max": 1e-12}
    if case["dtype"] == "f32":
        return {"rel": 5e-6, "max": 1e-4}
    if case["dtype"] == "tf32":
        return {"rel": 1e-4, "max": 5e-4}
    return {"rel": 7e-3, "max": 1.6e-2}


# ---- what run() computes, in 64 bits and without the kernels --------------------------------------------------------

E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def wrap(u):
    """A 64-bit constant as the signed number that torch's wrapping int64 arithmetic takes."""
    return u - (1 << 64) if u >> 63 else u


def mix64(z):
    """splitmix64's finaliser."""
    z = z + wrap(0x9E3779B97F4A7C15)
    z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * wrap(0xBF58476D1CE4E5B9)
    z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * wrap(0x94D049BB133111EB)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def fma(a, b, c):
    return (a.double() * b.double() + c).float()


def log_f32(x):
    """The generator's logarithm, one float32 operation after the other: x = m * 2^e, ln m = 2 atanh((m - 1) / (m + 1))."""
    m, e = torch.frexp(x)
    m, e = m * 2, e - 1
    high = m > 1.41421354
    m, e = torch.where(high, m * 0.5, m), torch.where(high, e + 1, e)
    t = (m - 1) / (m + 1)
    s = t * t
    p = torch.full_like(t, 1 / 11)
    for c in (1 / 9, 1 / 7, 1 / 5, 1 / 3, 1.0):
        p = fma(p, s, float(np.float32(c)))
    return fma(e.float(), torch.full_like(t, math.log(2)), (2 * t * p).double())


def cos_2pi_f32(u):
    q = u * 4
    k = q.to(torch.int32)
    th = (q - k) * 1.57079637
    s = th * th
    c, n = torch.full_like(s, -1 / math.factorial(14)), torch.full_like(s, -1 / math.factorial(15))
    for i in range(6, -1, -1):
        sign = -1.0 if i & 1 else 1.0
        c = fma(c, s, float(np.float32(sign / math.factorial(2 * i))))
        n = fma(n, s, float(np.float32(sign / math.factorial(2 * i + 1))))
    n = n * th
    return torch.where(k == 0, c, torch.where(k == 1, -n, torch.where(k == 2, -c, n)))


def normals(n, seed, wide=False):
    """clpk_fill_f32's N(0, 0.02): as the float32 values that it is defined by, or (wide) as the deviate itself in 64 bits."""
    base = int(mix64(torch.tensor(seed, dtype=torch.int64)))
    out = torch.empty(n, dtype=torch.float64 if wide else torch.float32, device="cuda")
    for at in range(0, n, 1 << 25):
        h = mix64(torch.arange(at, min(n, at + (1 << 25)), dtype=torch.int64, device="cuda") + base)
        u1, u2 = (((h >> 41) & 0x7FFFFF) + 1).double() / 2 ** 23, (h & 0xFFFFFF).double() / 2 ** 24
        if wide:
            v = 0.02 * torch.sqrt(-2 * torch.log(u1)) * torch.cos(2 * math.pi * u2)
        else:
            v = fma(torch.sqrt(-2 * log_f32(u1.float())) * cos_2pi_f32(u2.float()), torch.full_like(u1.float(), 0.02), 0.0)
        out[at:at + v.numel()] = v
    return out


def e2m1(x):
    """Nearest e2m1 value, ties to the even code: a tie goes up where the code below it is odd."""
    codes = torch.tensor(E2M1, device=x.device)
    code = torch.zeros(x.shape, dtype=torch.int64, device=x.device)
    for i in range(7):
        edge = (E2M1[i] + E2M1[i + 1]) / 2
        code += (x.abs() >= edge) if i & 1 else (x.abs() > edge)
    return codes[code].copysign(x)


def operand_f64(dtype, rows, cols, seed):
    """(the operand's decoded values in float64, its tensor scale)"""
    f = normals(rows * cols, seed)
    if dtype in ("f32", "f64"):
        return f.double().view(rows, cols), 1.0
    if dtype == "tf32":
        b = f.view(torch.int32)
        b = (b + 0xFFF + ((b >> 13) & 1)) & ~0x1FFF
        return b.view(torch.float32).double().view(rows, cols), 1.0
    plain = {"bf16": torch.bfloat16, "f16": torch.float16, "e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}
    if dtype in plain:
        return f.to(plain[dtype]).double().view(rows, cols), 1.0
    blocks = f.view(-1, SCALE_BLOCK[dtype])
    if dtype == "mxf4":
        scale = 1.0
        s = torch.ldexp(torch.ones_like(blocks[:, :1]), torch.frexp(blocks.abs().amax(1, keepdim=True))[1] - 3)
    else:
        scale = float(np.float32(f.abs().max().item()) / np.float32(6.0 * 448.0))
        blocks = blocks / torch.tensor(scale, dtype=torch.float32, device=f.device)
        s = (blocks.abs().amax(1, keepdim=True) / torch.tensor(6.0, device=f.device)).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    q = torch.where(s > 0, e2m1(blocks / s), torch.zeros_like(blocks))
    return (q.double() * s.double()).view(rows, cols), scale


def exact(case, seed):
    """The floating results in 64 bits: products of the operands as they are quantised, and the deviates behind the generated
    floats.  Whole-number products, bytes, and the streams' copies and sums have none."""
    if case["path"] == "operands" and case["dtype"] != "i8":
        out = {"f32": normals(case["rows"] * case["cols"], seed, wide=True)}
        if case["dtype"] != "f32":
            out["packed"] = None
        if case["dtype"] in SCALE_BLOCK:
            out.update(scales=None, tensor_scale=None)
        return out
    if case["path"] != "gemm" or case["dtype"] == "i8":
        return None
    dtype, m, n, k = case["dtype"], case["m"], case["n"], case["k"]
    a, scale_a = operand_f64(dtype, m, k, 2 * seed)
    b, scale_b = operand_f64("e4m3" if dtype == "e5m2" else dtype, n, k, 2 * seed + 1)
    c = a @ b.T
    c *= float(np.float32(np.float32(scale_a) * np.float32(scale_b)))
    return {"c": c, "status": None}
