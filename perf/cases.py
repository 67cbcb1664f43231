"""Performance cases of the B200 `cuda` provider (skb_cuda).

The cases are the calls a user of the library makes, through its device entry
points: the composed nonlinear flux in both of its forms, the plain and pruned
horizontal transforms, the grouped vertical GEMM, the spectral pipeline and the
type-I vertical transforms.  listed() holds fixed sizes, draw() further ones of
the same ranges; prepare() builds what a program holds before the call, run()
is one pass, work() what it cannot do without and exact() its result in 64-bit
arithmetic from plain torch.
"""

import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spectral-kernel-benchmarks_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import skb_cuda  # noqa: E402

FLUX_MODES = {"fp64": skb_cuda.FLUX_FP64_PLAIN, "fp32": skb_cuda.FLUX_FP32, "tf32x3": skb_cuda.FLUX_SPLIT_TF32X3,
              "bf16x3": skb_cuda.FLUX_SPLIT_BF16X3}
GEMM_MODES = {"fp64": skb_cuda.GEMM_FP64, "fp32": skb_cuda.GEMM_FP32, "tf32x3": skb_cuda.GEMM_TF32X3,
              "bf16x3": skb_cuda.GEMM_BF16X3}


def listed():
    return [
        # The headline run: an ensemble of eight 512^2 x 129 states per call, in
        # split precision, with the launch shapes autotuned as the benchmark does.
        {"name": "flux_split_512_ensemble", "kind": "flux", "n": 512, "nz": 129, "targets": 4, "members": 8,
         "mode": "tf32x3", "autotune": True},
        # A batch of the middle serving class, on a handle that nobody tuned.
        {"name": "flux_split_256_batch", "kind": "flux", "n": 256, "nz": 65, "targets": 3, "members": 4,
         "mode": "tf32x3", "autotune": False},
        # One request of the smallest serving class: latency and launches count.
        {"name": "flux_split_128_single", "kind": "flux", "n": 128, "nz": 33, "targets": 3, "members": 1,
         "mode": "tf32x3", "autotune": False},
        # The FP64 drop-in flux of one full-size state.
        {"name": "flux_fp64_512_single", "kind": "flux", "n": 512, "nz": 129, "targets": 4, "members": 1,
         "mode": "fp64", "autotune": False},
        # Plain FP64 2-D transform and back, the reference's first benchmark.
        {"name": "fft_fp64_256", "kind": "fft", "nx": 256, "ny": 256, "nz": 65, "fields": 3, "precision": "fp64"},
        # The same in FP32 on an oblong grid with a plane count that fills no block.
        {"name": "fft_fp32_oblong", "kind": "fft", "nx": 512, "ny": 128, "nz": 37, "fields": 5, "precision": "fp32"},
        # Zero-filled inverse and truncating forward transform of a whole
        # full-size state (four fields), the largest horizontal call.
        {"name": "pruned_fp64_512", "kind": "pruned", "nx": 512, "ny": 512, "nz": 129, "fields": 4,
         "precision": "fp64"},
        # The reference's pruned-horizontal benchmark in FP32.
        {"name": "pruned_fp32_256", "kind": "pruned", "nx": 256, "ny": 256, "nz": 65, "fields": 3,
         "precision": "fp32"},
        # The reference's vertical GEMM benchmark: 2,045 K^2 groups, FP64.
        {"name": "vertical_fp64_256", "kind": "vertical", "n": 256, "nz": 65, "fields": 3, "precision": "fp64"},
        # The tensor-core form with a ragged level count and more fields.
        {"name": "vertical_tf32x3_256", "kind": "vertical", "n": 256, "nz": 100, "fields": 4, "precision": "tf32x3"},
        # A whole spectral round trip (five stages) on a ragged small state.
        {"name": "pipeline_fp32_128", "kind": "pipeline", "n": 128, "nz": 50, "fields": 3, "precision": "fp32"},
        # Constant stratification: forward and inverse type-I transforms of the
        # three-channel arena of a 512^2 state's retained modes.
        {"name": "type1_fp64_129", "kind": "type1", "rows": 45765, "channels": 3, "nz": 129, "dst": False,
         "precision": "fp64"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["flux", "flux", "flux", "fft", "fft", "pruned", "pruned", "vertical", "vertical", "pipeline",
                       "type1"])
    while True:
        if kind == "flux":
            n = rng.choice([64, 128, 128, 256, 256, 512])
            mode = rng.choice(["tf32x3", "tf32x3", "tf32x3", "bf16x3", "fp64", "fp64", "fp32"])
            case = {"kind": kind, "n": n, "nz": rng.randint(13, 129), "targets": rng.choice([3, 4]),
                    "members": _log_int(rng, 1, 8), "mode": mode, "autotune": rng.random() < 0.25}
            small = n * n * case["nz"] * case["members"] <= (100e6 if mode in ("tf32x3", "bf16x3") else 40e6)
        elif kind in ("fft", "pruned"):
            case = {"kind": kind, "nx": rng.choice([64, 128, 256, 512, 1024]),
                    "ny": rng.choice([64, 128, 256, 512, 1024]), "nz": _log_int(rng, 1, 129),
                    "fields": rng.randint(1, 5), "precision": rng.choice(["fp64", "fp32"])}
            small = case["nx"] * case["ny"] * case["nz"] * case["fields"] <= 130e6
        elif kind in ("vertical", "pipeline"):
            case = {"kind": kind, "n": rng.choice([64, 128, 256]), "nz": rng.randint(13, 129),
                    "fields": rng.randint(1, 5),
                    "precision": rng.choice(["fp64", "fp64", "fp32", "tf32x3", "bf16x3"] if kind == "vertical"
                                            else ["fp64", "fp32"])}
            small = True
        else:
            case = {"kind": kind, "rows": _log_int(rng, 2000, 130000), "channels": rng.randint(1, 3),
                    "nz": rng.choice([33, 65, 129, 129, 257, rng.randint(20, 140)]), "dst": rng.random() < 0.5,
                    "precision": rng.choice(["fp64", "fp64", "fp32"])}
            small = case["rows"] * case["channels"] * case["nz"] <= 20e6
        if small:
            return case


# ---------------------------------------------------------------- geometry

def _nj(nz):
    return 2 * (nz - 1) // 3


class _Modes:
    """Retained modes of an Nx x Ny grid (radial 2/3 rule), ordered by radius,
    k and l, with the stored half-spectrum cell of each."""

    def __init__(self, nx, ny):
        k, l = np.meshgrid(np.arange(-(nx // 2) + 1, nx // 2), np.arange(-(ny // 2) + 1, ny // 2), indexing="xy")
        k, l = k.ravel(), l.ravel()
        radial = np.sqrt((2.0 * np.pi * k) ** 2 + (2.0 * np.pi * l) ** 2)
        held = ((l > 0) | ((l == 0) & (k >= 0))) & (radial <= 2.0 * (2.0 * np.pi * (nx // 2)) / 3.0)
        k, l, radial = k[held], l[held], radial[held]
        order = np.lexsort((l, k, radial))
        self.k, self.l = k[order], l[order]
        self.conj = self.k < 0
        self.kx = np.abs(self.k)
        self.ky = np.where(self.conj, -self.l, self.l) % ny
        self.partner = (self.kx == 0) & (self.ky != 0) & (2 * self.ky != ny)
        key = self.k ** 2 + self.l ** 2
        self.group = np.r_[0, np.cumsum(key[1:] != key[:-1])]
        self.keys = key[np.r_[True, key[1:] != key[:-1]]]

    def __len__(self):
        return len(self.k)


def _k2_matrices(modes, nz, device):
    """The K^2 pair-rotation operators: forward [group][j][z] (their transposes
    are the inverse ones)."""
    nj = _nj(nz)
    j, z = np.arange(nj)[:, None], np.arange(nz)[None, :]
    base = np.where(j == 0, np.sqrt(1.0 / nz), np.sqrt(2.0 / nz)) * np.cos(np.pi * (z + 0.5) * j / nz)
    phase = 0.5 * np.pi * (modes.keys % 4093 + 1) / 4094.0
    c, s = np.cos(phase)[:, None, None], np.sin(phase)[:, None, None]
    out = np.empty((len(modes.keys), nj, nz))
    pairs = nj // 2
    out[:, 0:2 * pairs:2] = c * base[0:2 * pairs:2] + s * base[1:2 * pairs:2]
    out[:, 1:2 * pairs:2] = -s * base[0:2 * pairs:2] + c * base[1:2 * pairs:2]
    if nj % 2:
        out[:, nj - 1] = np.where(modes.keys % 2 == 1, -1.0, 1.0)[:, None] * base[nj - 1]
    return torch.from_numpy(out).to(device)


# ----------------------------------------------------------------- prepare

_STREAM = None


def _stream():
    """The stream of the program's work (a torch stream; its handle goes to the library)."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM.cuda_stream


def _real(case):
    return torch.float64 if case.get("precision", case.get("mode")) == "fp64" else torch.float32


def _complex(case):
    return torch.complex128 if _real(case) == torch.float64 else torch.complex64


def _spectral(modes, shape, seed, dtype):
    """Complex Gaussian amplitudes with a k^-3 power-law fall-off (the kx = 0 mean is real)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, dtype=dtype, device="cuda", generator=g)
    decay = torch.from_numpy((1.0 + modes.k.astype(np.float64) ** 2 + modes.l.astype(np.float64) ** 2) ** -1.5)
    mode_axis = shape.index(len(modes))
    view = [1] * len(shape)
    view[mode_axis] = len(modes)
    x *= decay.to("cuda").to(torch.view_as_real(x).dtype).view(view)
    x.select(mode_axis, 0).imag.zero_()
    return x


def _uniform(shape, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape, dtype=dtype, device="cuda", generator=g).mul_(2.0).sub_(1.0)


def prepare(case, seed):
    kind = case["kind"]
    real, cplx = _real(case), _complex(case)
    if kind == "flux":
        n, nz, targets, members = case["n"], case["nz"], case["targets"], case["members"]
        modes = _Modes(n, n)
        modal = _spectral(modes, (members, len(modes), 3 + 3 * targets, _nj(nz)), seed, cplx)
        out = torch.zeros((members, len(modes), targets, _nj(nz)), dtype=cplx, device="cuda")
        flux = skb_cuda.Flux(n, nz, targets=targets, members=members, mode=FLUX_MODES[case["mode"]])
        torch.cuda.synchronize()
        if case["autotune"]:
            flux.autotune(modal.data_ptr(), out.data_ptr())
        return {"kind": kind, "flux": flux, "in": modal, "out": out, "stream": _stream()}
    if kind in ("fft", "pruned"):
        w = skb_cuda.Workload(case["nx"], case["ny"], case["nz"], case["fields"])
        precision = skb_cuda.FP64 if real == torch.float64 else skb_cuda.FP32
        if kind == "fft":
            field = _uniform((w.fields, w.nz, w.ny, w.nx), seed, real)
            return {"kind": kind, "fft": skb_cuda.FFTProvider(w, precision), "real": field,
                    "spectrum": torch.zeros((w.ny, w.nx_half, w.planes), dtype=cplx, device="cuda"),
                    "back": torch.zeros_like(field), "stream": _stream()}
        modes = _Modes(w.nx, w.ny)
        retained = _spectral(modes, (len(modes), w.fields, w.nz), seed, cplx)
        return {"kind": kind, "pruned": skb_cuda.PrunedProvider(w, precision), "retained": retained,
                "real": torch.zeros((w.fields, w.nz, w.ny, w.nx), dtype=real, device="cuda"),
                "back": torch.zeros_like(retained), "views": _views(retained), "stream": _stream()}
    if kind == "vertical":
        w = skb_cuda.Workload(case["n"], case["n"], case["nz"], case["fields"])
        modes = _Modes(w.nx, w.ny)
        forward, inverse, _ = skb_cuda.vertical_family(w)
        gemm = skb_cuda.VerticalGemmProvider(w, skb_cuda.squared_wavenumber_groups(w), forward, inverse,
                                             gemm_precision=GEMM_MODES[case["precision"]])
        physical = _spectral(modes, (len(modes), w.fields, w.nz), seed, cplx)
        return {"kind": kind, "gemm": gemm, "physical": physical,
                "modal": torch.zeros((len(modes), w.fields, w.nj), dtype=cplx, device="cuda"),
                "back": torch.zeros_like(physical), "stream": _stream()}
    if kind == "pipeline":
        w = skb_cuda.Workload(case["n"], case["n"], case["nz"], case["fields"])
        precision = skb_cuda.FP64 if real == torch.float64 else skb_cuda.FP32
        field = _uniform((w.fields, w.nz, w.ny, w.nx), seed, real)
        return {"kind": kind, "pipeline": skb_cuda.SpectralPipeline(w, precision), "real": field,
                "back": torch.zeros_like(field), "stream": _stream()}
    precision = skb_cuda.FP64 if real == torch.float64 else skb_cuda.FP32
    g = torch.Generator(device="cuda").manual_seed(seed)
    arena = torch.randn((case["rows"], case["channels"], case["nz"]), dtype=cplx, device="cuda", generator=g)
    return {"kind": kind, "plans": skb_cuda.ConstantStratificationVertical(case["rows"], case["nz"], precision),
            "arena": arena, "transform": skb_cuda.TYPE1_DST if case["dst"] else skb_cuda.TYPE1_DCT,
            "channels": case["channels"], "stream": _stream()}


def _views(retained):
    """Field views over a retained array [mode][field][z]."""
    modes, fields, nz = retained.shape
    return [(retained.data_ptr() + f * nz * retained.element_size(), None, fields * nz) for f in range(fields)]


# --------------------------------------------------------------------- run

def run(state):
    kind, stream = state["kind"], state["stream"]
    if kind == "flux":
        state["flux"].execute_device(state["in"].data_ptr(), state["out"].data_ptr(), stream)
        return state["out"]
    if kind == "fft":
        state["fft"].forward_device(state["real"].data_ptr(), state["spectrum"].data_ptr(), stream)
        state["fft"].inverse_device(state["spectrum"].data_ptr(), state["back"].data_ptr(), stream)
        return {"spectrum": state["spectrum"], "real": state["back"]}
    if kind == "pruned":
        state["pruned"].inverse_device(state["views"], state["real"].data_ptr(), stream)
        state["pruned"].forward_device(state["real"].data_ptr(), _views(state["back"]), 1.0, stream)
        return {"real": state["real"], "retained": state["back"]}
    if kind == "vertical":
        state["gemm"].forward_device(state["physical"].data_ptr(), None, state["modal"].data_ptr(), None, stream)
        state["gemm"].inverse_device(state["modal"].data_ptr(), None, state["back"].data_ptr(), None, stream)
        return {"modal": state["modal"], "physical": state["back"]}
    if kind == "pipeline":
        state["pipeline"].execute_device(state["real"].data_ptr(), state["back"].data_ptr(), stream)
        return state["back"]
    # Type-I transforms work in place: forward with the WVM normalisation, then inverse.
    for normalize in (True, False):
        state["plans"].transform_device(state["arena"].data_ptr(), state["transform"], state["channels"], 0,
                                        state["channels"], normalize, stream)
    return state["arena"]


# -------------------------------------------------------------------- work

def work(case):
    kind = case["kind"]
    es = 8 if _real(case) == torch.float64 else 4

    def fft2d(nx, ny, planes):
        return 2.5 * nx * ny * math.log2(nx * ny) * planes

    if kind == "flux":
        n, nz, t, members, nj = case["n"], case["nz"], case["targets"], case["members"], _nj(case["nz"])
        modes = _Modes(n, n)
        fields = 3 + 4 * t
        return {"bytes": 2 * es * members * len(modes) * fields * nj + 2 * es * len(modes.keys) * nz * nj,
                "flops": 4.0 * members * len(modes) * fields * nj * nz + members * fft2d(n, n, fields * nz)
                + 6.0 * members * t * n * n * nz}
    if kind == "fft":
        planes = case["nz"] * case["fields"]
        spectrum = 2 * es * case["ny"] * (case["nx"] // 2 + 1) * planes
        return {"bytes": 2 * (es * case["nx"] * case["ny"] * planes + spectrum),
                "flops": 2 * fft2d(case["nx"], case["ny"], planes)}
    if kind == "pruned":
        planes = case["nz"] * case["fields"]
        retained = 2 * es * len(_Modes(case["nx"], case["ny"])) * planes
        return {"bytes": 2 * (es * case["nx"] * case["ny"] * planes + retained),
                "flops": 2 * fft2d(case["nx"], case["ny"], planes)}
    if kind == "type1":
        values = case["rows"] * case["channels"] * case["nz"]
        return {"bytes": 2 * 2 * 2 * es * values, "flops": 2 * 5.0 * values * math.log2(2 * (case["nz"] - 1))}
    modes = _Modes(case["n"], case["n"])
    nz, nj, columns = case["nz"], _nj(case["nz"]), len(modes) * case["fields"]
    gemm = 2 * 4.0 * columns * nj * nz
    matrices = 2 * es * len(modes.keys) * nz * nj
    if kind == "vertical":
        return {"bytes": 2 * 2 * es * columns * (nz + nj) + matrices, "flops": gemm}
    planes = nz * case["fields"]
    return {"bytes": 2 * es * case["n"] ** 2 * planes + matrices,
            "flops": gemm + 2 * fft2d(case["n"], case["n"], planes)}


# ------------------------------------------------------------------- exact

def _embed(modes, retained, nx, ny):
    """Retained values [mode][plane] -> half spectra [plane][ky][kx], zero elsewhere."""
    kx, ky = (torch.from_numpy(a).to(retained.device) for a in (modes.kx, modes.ky))
    conj = torch.from_numpy(modes.conj).to(retained.device)[:, None]
    stored = torch.where(conj, retained.conj(), retained)
    cells = torch.zeros((ny * (nx // 2 + 1), retained.shape[1]), dtype=retained.dtype, device=retained.device)
    cells[ky * (nx // 2 + 1) + kx] = stored
    rep = torch.from_numpy(modes.partner).to(retained.device)
    cells[(ny - ky[rep]) * (nx // 2 + 1)] = stored[rep].conj()
    return cells.t().reshape(-1, ny, nx // 2 + 1)


def _gather(modes, spectra):
    """Half spectra [plane][ky][kx] -> retained values [mode][plane]."""
    kx, ky = (torch.from_numpy(a).to(spectra.device) for a in (modes.kx, modes.ky))
    values = spectra[:, ky, kx].t()
    return torch.where(torch.from_numpy(modes.conj).to(spectra.device)[:, None], values.conj(), values)


def _c2r(spectra, nx, ny):
    """Unnormalised inverse transform of half spectra [plane][ky][kx]."""
    rows = torch.fft.ifft(spectra, dim=1, norm="forward")
    rows[:, :, 0].imag.zero_()
    rows[:, :, nx // 2].imag.zero_()
    return torch.fft.irfft(rows, n=nx, dim=2, norm="forward")


def _vertical(matrices, group, x, transpose):
    """Apply each mode's group operator to x [mode][field][i]."""
    out = []
    for a in range(0, x.shape[0], 8192):
        m = matrices[group[a:a + 8192]]
        v = torch.view_as_real(x[a:a + 8192]).permute(0, 2, 1, 3).reshape(m.shape[0], x.shape[2], -1)
        y = torch.bmm(m.transpose(1, 2) if transpose else m, v)
        y = y.reshape(y.shape[0], y.shape[1], x.shape[1], 2).permute(0, 2, 1, 3).contiguous()
        out.append(torch.view_as_complex(y))
    return torch.cat(out)


def exact(case, seed):
    """run()'s outputs in 64-bit arithmetic."""
    kind = case["kind"]
    cplx = _complex(case)
    if kind == "flux":
        n, nz, targets, members = case["n"], case["nz"], case["targets"], case["members"]
        modes = _Modes(n, n)
        group = torch.from_numpy(modes.group).to("cuda")
        matrices = _k2_matrices(modes, nz, "cuda")
        modal = _spectral(modes, (members, len(modes), 3 + 3 * targets, _nj(nz)), seed, cplx)
        out = torch.empty((members, len(modes), targets, _nj(nz)), dtype=torch.complex128, device="cuda")
        for m in range(members):
            physical = _vertical(matrices, group, modal[m].to(torch.complex128), True)

            def volume(f):
                return _c2r(_embed(modes, physical[:, f], n, n), n, n)

            velocity = [volume(f) for f in range(3)]
            products = []
            for t in range(targets):
                p = sum(velocity[i] * volume(3 + 3 * t + i) for i in range(3)) * (-1.0 / float(n) ** 4)
                products.append(_gather(modes, torch.fft.rfft2(p)))
            out[m] = _vertical(matrices, group, torch.stack(products, 1), False)
        return out
    if kind == "fft":
        nx, ny, planes = case["nx"], case["ny"], case["nz"] * case["fields"]
        field = _uniform((case["fields"], case["nz"], ny, nx), seed, _real(case)).to(torch.float64)
        spectrum = torch.fft.rfft2(field.reshape(planes, ny, nx)).permute(1, 2, 0).contiguous()
        return {"spectrum": spectrum, "real": field * float(nx * ny)}
    if kind == "pruned":
        nx, ny, nz, fields = case["nx"], case["ny"], case["nz"], case["fields"]
        modes = _Modes(nx, ny)
        retained = _spectral(modes, (len(modes), fields, nz), seed, cplx).to(torch.complex128)
        field = torch.empty((fields, nz, ny, nx), dtype=torch.float64, device="cuda")
        for f in range(fields):
            field[f] = _c2r(_embed(modes, retained[:, f], nx, ny), nx, ny)
        return {"real": field, "retained": retained * float(nx * ny)}
    if kind == "type1":
        rows, channels, nz = case["rows"], case["channels"], case["nz"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn((rows, channels, nz), dtype=cplx, device="cuda", generator=g).to(torch.complex128)
        m = nz - 1
        if case["dst"]:
            # Normalised forward (endpoints zeroed), then inverse over the interior.
            x[..., 0], x[..., m] = 0.0, 0.0
            return x * 2.0

        def dct(v):
            return torch.fft.fft(torch.cat([v, v[..., 1:m].flip(-1)], -1), dim=-1)[..., :nz]

        y = dct(x) / m
        y[..., m] *= 0.5
        return dct(y)
    n, nz, fields = case["n"], case["nz"], case["fields"]
    modes = _Modes(n, n)
    group = torch.from_numpy(modes.group).to("cuda")
    matrices = _k2_matrices(modes, nz, "cuda")
    if kind == "vertical":
        physical = _spectral(modes, (len(modes), fields, nz), seed, cplx).to(torch.complex128)
        modal = _vertical(matrices, group, physical, False)
        return {"modal": modal, "physical": _vertical(matrices, group, modal, True)}
    field = _uniform((fields, nz, n, n), seed, _real(case)).to(torch.float64)
    retained = _gather(modes, torch.fft.rfft2(field.reshape(fields * nz, n, n))).reshape(len(modes), fields, nz)
    modal = _vertical(matrices, group, retained, False)
    j = np.arange(_nj(nz))[None, None, :]
    f = np.arange(fields)[None, :, None]
    key = (17 * np.abs(modes.k)[:, None, None] + 29 * np.abs(modes.l)[:, None, None] + 7 * j + 11 * f) % 97
    modal = modal * torch.from_numpy(0.75 + 0.5 * key / 96.0).to("cuda")
    retained = _vertical(matrices, group, modal, True).reshape(len(modes), fields * nz)
    return _c2r(_embed(modes, retained, n, n), n, n).reshape(fields, nz, n, n)
