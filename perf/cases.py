"""Timing cases of the spectrometer over the sizes it is used at.

A case names an entry point and a configuration:

  kind "resident"  rawspec_start_processing on input that is already on the GPU (a producer on the same
                   GPU, or blocks copied ahead of time); a pass is the buffers of one integration, from
                   the wait for the previous dumps to the dumps in host memory
  kind "stream"    the command line client's loop from pinned host blocks: wait_for_completion, then
                   copy_blocks_to_gpu_and_start_processing, per buffer
  kind "group"     one buffer each of several contexts through rawspec_gb300_start_processing_group
  kind "device"    rawspec_gb300_product_noalloc between two tensors of the caller

`products` lists "FFT length x spectra per integration" of each output product, `npol` their Npolout.
"""
import ctypes as C
import math

import numpy as np
import torch

from rawspec_gb300 import api

MIB = 1 << 20


def listed():
    base = dict(npols=2, nbits=8, nant=1, conj=False, inverse=False, npol=1, nb=1, contexts=1)

    def case(name, **kw):
        return {"name": name, **base, **kw}

    return [
        # The smallest plain configuration: eight channels of one recorder, one 2 MiB block at a time;
        # a buffer is little more than its launches and the dump.
        case("small_1024", kind="resident", nc=8, ntpb=65536, products="1024x16"),
        # A pipeline that owns its GPU memory asks for one short integration of a few channels: the
        # smallest call there is.
        case("device_small_256", kind="device", nc=5, ntpb=6912, npol=4, products="256x9"),
        # The same entry point on a large 16-bit buffer, Stokes parameters, an odd number of channels.
        case("device_16bit_2048", kind="device", nc=45, ntpb=786432, nbits=16, npol=-4, products="2048x24"),
        # The production shape of the command line client: 64 channels, high-resolution (2^20 points),
        # high-time-resolution (8) and mid (1024) products of every 256 MiB buffer, the whole 51-buffer
        # integration with its dumps.
        case("production_total_power", kind="resident", nc=64, ntpb=524288, nb=2,
             products="1048576x51,8x128,1024x3072"),
        # The same three products with the cross terms kept (XX, YY, Re XY, Im XY), half the band.
        case("production_full_pol", kind="resident", nc=32, ntpb=524288, nb=2, npol=4,
             products="1048576x51,8x128,1024x3072"),
        # The production shape as the client runs it, every buffer copied from host blocks.
        case("production_stream", kind="stream", nc=64, ntpb=524288, nb=2, products="1048576x51,8x128,1024x3072"),
        # Four antennas, 4-bit samples, Stokes spectra and their weighted incoherent sum.
        case("antennas_4bit_stokes", kind="stream", nc=64, ntpb=262144, nbits=4, nant=4, npol=-4,
             products="4096x64,64x1024"),
        # Medium-resolution spectra, several of them integrated within one buffer (the serving mix's 65536).
        case("spectra_65536", kind="resident", nc=32, ntpb=262144, nb=4, products="65536x16"),
        # A 16-bit recorder of one polarisation, an odd number of channels, input of the other sideband.
        case("zoom_16bit_one_pol", kind="resident", nc=21, npols=1, ntpb=262144, nb=2, nbits=16, conj=True,
             inverse=True, products="16384x8"),
        # Four short products of one small recorder at once, cross terms kept.
        case("short_products_full_pol", kind="resident", nc=8, ntpb=65536, nb=16, npol=4,
             products="4096x256,1024x512,256x256,8x128"),
        # Buffers of eight small observations that arrive together (the job server's shared launches).
        case("group_of_eight", kind="group", nc=8, ntpb=262144, contexts=8, products="512x64"),
        # One very long transform of a few channels: the finest resolution, four buffers an integration.
        case("finest_4194304", kind="resident", nc=5, ntpb=1048576, nb=4, npol=-4, products="4194304x4"),
    ]


def _divisors(n):
    return [d for d in range(1, min(n, 1 << 14) + 1) if n % d == 0]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["resident"] * 4 + ["stream"] * 3 + ["device"] * 2 + ["group"])
    npols = rng.choice([2, 2, 2, 1])
    nbits = rng.choice([8, 8, 8, 16] if kind in ("device", "group") else [8, 8, 8, 4, 16])
    npol = rng.choice([1, 1, 4, -4]) if npols == 2 else 1
    planes = abs(npol)
    contexts = rng.randint(2, 8) if kind == "group" else 1
    longest = 12 if kind in ("device", "group") else 22
    n = 1 << (rng.randint(3, 12) if rng.random() < 0.5 else rng.randint(3, longest))
    nc = _log_int(rng, 1, 64)
    nant = 1
    if kind in ("resident", "stream") and nc > 1 and rng.random() < 0.25:
        nant = rng.randint(2, 4)
        nc = max(1, nc // nant) * nant
    word = npols * max(1, 2 * nbits // 8)  # bytes of a sample of all polarisations on the GPU
    least = max(64 << 10, nc * n * word)
    most = (256 if kind in ("resident", "stream") else 64) * MIB
    while nc > nant and nc * n * max(word, planes * 2) > most:
        nc = max(1, nc // nant // 2) * nant
    size = _log_int(rng, min(least, most), most)
    s = max(1, size // (nc * n * word))  # spectra of the longest product in a buffer
    if s > 4 and rng.random() < 0.7:  # mostly counts with factors, odd ones among them
        f = rng.choice([2, 3, 4, 6, 8, 12, 16])
        s = max(1, s // f) * f if s >= f else s
    total = s * n
    nb = rng.choice([b for b in (1, 2, 3, 4, 8) if total % b == 0]) if kind in ("resident", "stream") else 1
    # the longest product: within the buffer, or over up to four buffers
    if kind in ("resident", "stream") and (s <= 4 or rng.random() < 0.25):
        na = s * rng.randint(1, 4)
    else:
        na = rng.choice([d for d in _divisors(s) if d * 16 >= min(s, 64)] or [s])
    products = [(n, na)]
    if kind in ("resident", "stream") and n >= 256 and rng.random() < 0.5:
        m = n >> rng.randint(2, (n.bit_length() - 1) - 3)
        sm = total // m
        products.append((m, rng.choice([d for d in _divisors(sm) if 16 <= d <= 4096] or [sm])))
    # dumps are a fraction of the input: integrate further where they are not
    for i, (m, a) in enumerate(products):
        sm = total // m
        if a < sm and sm // a * m * nc * planes * 4 > nc * total * word:
            products[i] = (m, sm)
    return dict(kind=kind, nc=nc, npols=npols, ntpb=total // nb, nb=nb, nbits=nbits, nant=nant, npol=npol,
                conj=rng.random() < 0.3, inverse=rng.random() < 0.2, contexts=contexts,
                products=",".join("%dx%d" % p for p in products))


def _products(case):
    return [tuple(int(v) for v in p.split("x")) for p in case["products"].split(",")]


def _buffers(case):
    """Buffers of a pass: every product's integration ends with the last one."""
    total = case["ntpb"] * case["nb"]
    count = 1
    for n, na in _products(case):
        count = math.lcm(count, max(1, na // (total // n)))
    return count


def _voltages(case, seed):
    """One buffer's codes on the GPU, [channel][time][pol][re, im]: complex Gaussian noise (sigma 20, or 2500
    in 16 bits; 4 bits: uniform with a gain for each antenna), rounded and clipped."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nc, total, nbits = case["nc"], case["ntpb"] * case["nb"], case["nbits"]
    out = torch.empty((nc, total, case["npols"], 2), dtype=torch.int16 if nbits == 16 else torch.int8, device="cuda")
    per_ant = nc // case["nant"]
    for c in range(nc):
        if nbits == 4:
            gain = 0.5 + 1.5 * ((c // per_ant) * 0.37 % 1.0)
            v = torch.rand(out.shape[1:], generator=g, device="cuda").mul_(16).sub_(8).mul_(gain).floor_().clamp_(-8, 7)
        else:
            v = torch.randn(out.shape[1:], generator=g, device="cuda").mul_(2500.0 if nbits == 16 else 20.0)
            lim = 1 << (nbits - 1)
            v.round_().clamp_(-lim, lim - 1)
        out[c] = v.to(out.dtype)
    return out


def _weights(case):
    return [0.5 + (0.618 * a) % 1.0 for a in range(case["nant"])]


def _fill(spec, case, codes):
    """The buffer's codes as the recorder's blocks, in the context's pinned host blocks."""
    for b in range(case["nb"]):
        blk = codes[:, b * case["ntpb"]:(b + 1) * case["ntpb"]]
        if case["nbits"] == 4:
            blk = ((blk[..., 0] & 15) << 4) | (blk[..., 1] & 15)
        raw = blk.contiguous().view(torch.uint8).reshape(-1)
        torch.from_numpy(spec.host_block(b))[: raw.numel()].copy_(raw)


def _dump_view(spec, pointer, floats):
    """A dump buffer as an array that keeps its context open."""
    class Buffer(C.c_float * floats):
        pass
    buf = Buffer.from_address(C.cast(pointer, C.c_void_p).value)
    buf.spec = spec
    return np.frombuffer(buf, dtype=np.float32)


def _outputs(spec, case):
    out = []
    for i in range(len(_products(case))):
        floats = spec.ctx.h_pwrbuf_size[i] // 4
        out.append(_dump_view(spec, spec.ctx.h_pwrbuf[i], floats))
        if case["nant"] > 1:
            out.append(_dump_view(spec, spec.ctx.h_icsbuf[i], floats // case["nant"]))
    return out


def _noalloc():
    f = api.load_library().rawspec_gb300_product_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_uint, C.c_uint, C.c_uint, C.c_ulonglong, C.c_uint, C.c_uint, C.c_int, C.c_int, C.c_int,
                  C.c_void_p, C.c_void_p]
    return f


def prepare(case, seed):
    prods = [(n, na, case["npol"]) for n, na in _products(case)]
    state = {"case": case, "dir": -1 if case["inverse"] else 1}
    if case["kind"] == "device":
        n, na, npol = prods[0]
        state["in"] = _voltages(case, seed)
        state["out"] = torch.empty(case["ntpb"] // (n * na) * abs(npol) * case["nc"] * n, dtype=torch.float32,
                                   device="cuda")
        state["call"] = _noalloc()
        state["args"] = (case["nc"], case["npols"], case["nbits"], case["ntpb"], n, na, npol, state["dir"],
                         int(case["conj"]))
        return state
    specs = []
    for k in range(case["contexts"]):
        spec = api.Spectrometer(case["nc"], case["npols"], case["ntpb"], case["nbits"], prods, Nant=case["nant"],
                                Nb=case["nb"], conj=int(case["conj"]), collect=False,
                                weights=_weights(case) if case["nant"] > 1 else None)
        _fill(spec, case, _voltages(case, seed + 7919 * k))
        spec.copy_to_gpu()
        specs.append(spec)
    state["specs"] = specs
    state["outs"] = [_outputs(spec, case) for spec in specs]
    state["buffers"] = _buffers(case)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "device":
        rc = state["call"](state["in"].data_ptr(), *state["args"], state["out"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("rawspec_gb300_product_noalloc failed")
        return state["out"]
    specs, fft_dir = state["specs"], state["dir"]
    if kind == "stream":
        for _ in range(state["buffers"]):
            if specs[0].wait():
                raise RuntimeError("wait_for_completion failed")
            specs[0].copy_and_start(fft_dir)
    else:
        for spec in specs:
            if spec.wait():
                raise RuntimeError("wait_for_completion failed")
        for _ in range(state["buffers"]):
            if kind == "group":
                api.start_group(specs, [fft_dir] * len(specs))
            else:
                specs[0].start(fft_dir)
    return state["outs"]


def _dump_floats(case):
    total = case["ntpb"] * case["nb"]
    floats = 0
    for n, na in _products(case):
        one = max(1, total // (n * na)) * abs(case["npol"]) * case["nc"] * n
        floats += one + (one // case["nant"] if case["nant"] > 1 else 0)
    return floats


def work(case):
    total = case["ntpb"] * case["nb"]
    buffers = _buffers(case)
    samples = case["nc"] * total * case["npols"] * buffers * case["contexts"]
    flops = 0.0
    for n, _ in _products(case):
        flops += samples * (5.0 * math.log2(n) + 4)
    return {"bytes": samples * 2 * case["nbits"] / 8 + 4.0 * _dump_floats(case) * case["contexts"], "flops": flops}


def _exact_one(case, codes):
    """One context's outputs in 64 bits: every channel's spectra, detected, integrated, shifted."""
    total, npol = case["ntpb"] * case["nb"], case["npol"]
    lim = 32767 if case["nbits"] == 16 else 127
    sign = -1.0 if case["conj"] else 1.0
    outs = []
    for n, na in _products(case):
        nss = total // n
        nd = max(1, nss // na)
        nis = max(1, na // nss)
        res = np.empty((nd, abs(npol), case["nc"], n))
        for c in range(case["nc"]):
            x = codes[c].to(torch.float64).clamp_(-lim, lim).div_(lim)
            x = torch.complex(x[..., 0], x[..., 1]).t().reshape(case["npols"], nss, n)
            x = torch.fft.fft(x) if not case["inverse"] else torch.fft.ifft(x, norm="forward")
            p = x.real.square() + x.imag.square()
            if npol == 1:
                planes = [p.sum(0)]
            else:
                cross = x[0] * x[1].conj()
                first = [p[0], p[1]] if npol == 4 else [p[0] + p[1], p[0] - p[1]]
                planes = first + [cross.real, sign * cross.imag]
            acc = torch.stack([q.reshape(nd, -1, n).sum(1) for q in planes], 1) * nis
            res[:, :, c] = torch.fft.fftshift(acc, dim=-1).cpu().numpy()
        outs.append(res.reshape(-1))
        if case["nant"] > 1:
            w = np.array(_weights(case), dtype=np.float32).astype(np.float64)
            per = res.reshape(nd, abs(npol), case["nant"], -1, n)
            outs.append(np.einsum("dpacn,a->dpcn", per, w).reshape(-1))
    return outs


def exact(case, seed):
    if case["kind"] == "device":
        return torch.from_numpy(_exact_one(case, _voltages(case, seed))[0])
    return [_exact_one(case, _voltages(case, seed + 7919 * k)) for k in range(case["contexts"])]
