"""The calls that a program makes of this package, at the sizes it makes them: what the performance work is measured on.

Every case is one pass through the public module (`create_ffno3d`, `FFNO3D.forward`, its input gradient, its forward
mode) on inputs that are already on the GPU. A case names a direction, a model and a cube:

  predict  the forward pass of a synthesis or a served PREDICT request
  vjp      forward and input gradient, an inversion step (`heights`: the gradient in the heights too)
  jvp      the forward-mode derivative along an input tangent

Most models here have one or two blocks: a block is the unit of the network, and the calls of a deeper model repeat it.
Inputs have the distributions of the MULTI3D/Bifrost atmospheres that the network takes, normalised as it takes them.
"""
import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from ffnoml_gb300 import create_ffno3d

SPACING = 48e3      # horizontal spacing in metres
REFERENCE_LENGTH, FEATURE_WAVELENGTH, RANK, HIDDEN = 40.0, 0.3, 8, 128
MEAN_X = (4.75, 0.0, 0.0, 0.0, 17.5, -8.0)
STD_X = (2.5 / math.sqrt(12), 5.0, 5.0, 5.0, 7.0 / math.sqrt(12), 8.0 / math.sqrt(12))


def _case(name, kind, precision, width, layers, modes, atoms, shape, columns=False, heights=False):
    D, H, W = shape
    return dict(name=name, kind=kind, precision=precision, width=width, layers=layers, modes=modes, atoms=atoms, D=D,
                H=H, W=W, columns=columns, heights=heights)


def listed():
    return [
        # the smallest: the plain drop-in's forward of the small configuration (width 32, 4 blocks, M = 16, H)
        _case("predict_w32_fp32", "predict", "fp32", 32, 4, 16, "H", (64, 32, 32)),
        # the smallest and an ordinary served request: the whole width-64, 8-block, two-atom model in BF16
        _case("predict_served_small_bf16", "predict", "bf16", 64, 8, 32, "H,CA", (128, 32, 32)),
        _case("predict_served_bf16", "predict", "bf16", 64, 8, 32, "H,CA", (192, 64, 64)),
        # the largest cube of the benchmark configuration, forward only
        _case("predict_large_bf16", "predict", "bf16", 64, 2, 32, "H,CA", (256, 128, 128)),
        # an inversion step on the differentiation configuration's cube
        _case("vjp_bf16", "vjp", "bf16", 64, 2, 32, "H,CA", (256, 96, 96)),
        # a cut-out of a simulation box: no size a power of two, an odd plane
        _case("vjp_odd_bf16", "vjp", "bf16", 64, 1, 32, "H,CA", (101, 45, 75)),
        # the production network (width 96, M = 1001): its inversion step, and the plain drop-in's forward of a cut-out
        _case("vjp_w96_bf16", "vjp", "bf16", 96, 1, 1001, "H", (256, 64, 64)),
        _case("predict_w96_odd_fp32", "predict", "fp32", 96, 1, 1001, "H", (97, 61, 50)),
        # an atmosphere whose columns have their own height grids (hydrostatic heights)
        _case("vjp_columns_bf16", "vjp", "bf16", 64, 1, 32, "H,CA", (128, 48, 40), columns=True),
        # the plain FP32 drop-in, forward and inversion step (features and heights)
        _case("predict_large_fp32", "predict", "fp32", 64, 1, 32, "H,CA", (256, 128, 128)),
        _case("vjp_fp32", "vjp", "fp32", 64, 2, 32, "H,CA", (128, 64, 64), heights=True),
        # the forward-mode derivative (FP32 whatever the precision)
        _case("jvp_fp32", "jvp", "fp32", 64, 2, 32, "H,CA", (64, 48, 48)),
    ]


def _cost(c):
    """About the device time of a pass: voxels x blocks, weighted by direction, precision and width."""
    per = {"predict": 1.0, "vjp": 2.6, "jvp": 2.4}[c["kind"]] * (c["width"] / 64) ** 1.5
    per *= 6.5 if c["precision"] == "fp32" or c["kind"] == "jvp" else 1.0
    return c["D"] * c["H"] * c["W"] * (c["layers"] + 0.3) * per


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["predict", "predict", "predict", "vjp", "vjp", "vjp", "jvp"])
        precision = "fp32" if kind == "jvp" else rng.choice(["bf16", "bf16", "fp32"])
        width, modes, atoms = rng.choice([(32, 16, "H"), (64, 32, "H,CA"), (64, 32, "H,CA"), (64, 32, "H,CA"),
                                          (96, 1001, "H")])
        layers = rng.choice([1, 2, 4, 8]) if kind == "predict" and precision == "bf16" else rng.choice([1, 2])
        columns = kind == "vjp" and width < 96 and rng.random() < 0.2
        D = _log_int(rng, 48, 256)
        if columns:
            H, W = _log_int(rng, 16, 56), _log_int(rng, 16, 56)
        else:
            H, W = _log_int(rng, 20, 128), _log_int(rng, 20, 128)
        c = _case("", kind, precision, width, layers, modes, atoms, (D, H, W), columns=columns,
                  heights=kind == "vjp" and precision == "fp32")
        del c["name"]
        if _cost(c) <= limit:
            return c


# ---------------------------------------------------------------------------------------------------------- inputs
_MODELS = {}


def _model(c):
    """The network of a case, as a program holds it: built and moved to the GPU once, used for every cube."""
    key = (c["precision"], c["width"], c["layers"], c["modes"], c["atoms"])
    if key not in _MODELS:
        torch.manual_seed(7)
        atoms = c["atoms"].split(",")
        levels = 6 * len(atoms)
        m = create_ffno3d(6, levels, atoms=atoms, width=c["width"], n_layers=c["layers"],
                          z_min_wavelength=REFERENCE_LENGTH / (c["modes"] - 1))
        with torch.no_grad():       # the parts that a new network starts at zero, as a trained one has them
            for name, p in m.named_parameters():
                if ".freq_u." in name:
                    p.normal_(0.0, 0.1)
            at = 0
            for n in m.species_levels:
                m.proj2.weight[at + n].normal_(0.0, 0.3)
                m.proj2.bias[at + n].normal_(0.0, 0.3)
                at += n + 1
        m.set_normalization(MEAN_X, STD_X, torch.zeros(levels), torch.ones(levels))
        for p in m.parameters():    # inference: the inversion differentiates the inputs only
            p.requires_grad_(False)
        _MODELS[key] = m.cuda().eval().set_precision(c["precision"])
    return _MODELS[key]


def _heights(c):
    """Heights [1, D, H, W] in Mm from 14 down to -1; with columns, each column's grid stretched and shifted."""
    D, H, W = c["D"], c["H"], c["W"]
    z = torch.linspace(14.0, -1.0, D, device="cuda")[None, :, None, None].expand(1, D, H, W)
    if c["columns"]:
        h = torch.arange(H, device="cuda", dtype=torch.float32)[:, None]
        w = torch.arange(W, device="cuda", dtype=torch.float32)[None, :]
        z = z * (1.0 + 0.02 * torch.sin(0.37 * h + 0.23 * w)) + 0.05 * torch.cos(0.11 * h - 0.19 * w)
    return z.contiguous()


def _inputs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)
    D, H, W = c["D"], c["H"], c["W"]
    uniform = lambda lo, hi: lo + (hi - lo) * torch.rand(D, H, W, generator=g, device="cuda")
    normal = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x = torch.stack([uniform(3.5, 6.0), 5.0 * normal(D, H, W), 5.0 * normal(D, H, W), 5.0 * normal(D, H, W),
                     uniform(14.0, 21.0), uniform(-12.0, -4.0)])
    mean, std = (torch.tensor(v, device="cuda")[:, None, None, None] for v in (MEAN_X, STD_X))
    x = ((x - mean) / std)[None].contiguous()
    out = 6 * len(c["atoms"].split(","))
    more = None
    if c["kind"] == "vjp":
        more = normal(1, out, D, H, W)
    elif c["kind"] == "jvp":
        more = normal(1, 6, D, H, W)
    return x, _heights(c), more


def prepare(case, seed):
    x, z, more = _inputs(case, seed)
    if case["kind"] == "vjp":
        x.requires_grad_(True)
        z.requires_grad_(case["heights"])
    return {"case": case, "model": _model(case), "x": x, "z": z, "more": more}


def run(state):
    c, m, x, z = state["case"], state["model"], state["x"], state["z"]
    if c["kind"] == "predict":
        with torch.no_grad():
            return m(x, z, SPACING, SPACING)
    if c["kind"] == "vjp":
        y = m(x, z, SPACING, SPACING)
        grads = torch.autograd.grad(y, (x, z) if c["heights"] else (x,), state["more"])
        return [y.detach(), *grads]
    import torch.autograd.forward_ad as forward_ad
    with torch.no_grad(), forward_ad.dual_level():
        y = m(forward_ad.make_dual(x, state["more"]), z, SPACING, SPACING)
        return list(forward_ad.unpack_dual(y))


def _live_modes(c):
    """Height modes below the Nyquist wavenumber of the column (the taper is zero above it)."""
    spacing = 15.0 * (1.02 if c["columns"] else 1.0) / (c["D"] - 1)
    return min(c["modes"], int(REFERENCE_LENGTH / (2 * spacing)) + 1)


def work(case):
    D, H, W, C, n = case["D"], case["H"], case["W"], case["width"], case["layers"]
    V, M, species = D * H * W, _live_modes(case), len(case["atoms"].split(","))
    out, spectrum = 6 * species, (W // 2 + 1) / W
    mix = 4 * C * C + 4 * RANK * C
    # multiply-adds a voxel: the 1x1x1 convolutions, both mixings, the two height transforms, lift and projection; the
    # horizontal transforms as FFTs: 2.5 n log2 n operations for a real plane of n points, each way
    block = 31 * C * C + C + mix * spectrum + 4 * M * C + mix * M / D
    flops = 2 * V * (n * block + 6 * C + 2 * C * C + 2 * C * (out + species))
    flops += n * 5 * V * C * math.log2(H * W)
    values = V * (6 + 1 + out)
    if case["kind"] == "vjp":
        flops *= 2
        values += V * (out + 6 + (1 if case["heights"] else 0))
    elif case["kind"] == "jvp":
        flops *= 2
        values += V * (6 + out)
    weights = n * (31 * C * C + 13 * C) + 2 * C * C + 6 * C + 2 * C * (out + species)
    return {"bytes": 4 * (values + weights), "flops": flops}


# ----------------------------------------------------------------------------------- the same in 64 bits, plain torch
# ln of g / g_1, excitation energies in eV and ionisation stages of the two atoms' levels
_ATOMS = {"H": ([2.0, 8.0, 18.0, 32.0, 50.0, 1.0], [1, 1, 1, 1, 1, 2],
                [0.0, 10.198673740091325, 12.087318311066094, 12.748311674749516, 13.054262568222963,
                 13.60794573029334], math.log10(2.2697e-27)),
          "CA": ([2.0, 4.0, 6.0, 2.0, 4.0, 1.0], [2, 2, 2, 2, 2, 3],
                 [0.0, 1.69242903005873, 1.6999489817497997, 3.12337806212316, 3.151018087686871,
                  11.87181686885173], math.log10(1.0375e-21))}
_E, _K, _PLANCK, _MASS, _PI = 1.602189e-12, 1.380662e-16, 6.626176e-27, 9.109534e-28, 3.14159265359


class _Exact:
    """The network on one cube in double precision, channels last."""

    def __init__(self, c, z):
        self.c = c
        self.p = {k: v.detach().double() for k, v in _model(c).state_dict().items()}
        self.C = c["width"]
        # each level's share of its column, mean 1
        gap = 0.5 * (z[1:] - z[:-1]).abs()
        share = F.pad(gap, (0, 0, 0, 0, 0, 1)) + F.pad(gap, (0, 0, 0, 0, 1, 0))
        self.share = (share / share.mean(0, keepdim=True).clamp_min(1e-12))[..., None]
        self.z = z
        self.low = z - z.amin(0, keepdim=True)

    def mlp(self, a, first, second, x):
        return F.gelu(x @ self.p[a + first][:, :, 0, 0, 0].T) @ self.p[a + second][:, :, 0, 0, 0].T

    def norm(self, name, x):
        D, H, W, C = x.shape
        g = x.reshape(D, H, W, 8, C // 8)
        w = self.share[..., None]
        total = w.sum() * (C // 8)
        mean = (w * g).sum((0, 1, 2, 4), keepdim=True) / total
        var = (w * (g - mean) ** 2).sum((0, 1, 2, 4), keepdim=True) / total
        y = ((g - mean) * torch.rsqrt(var + 1e-5)).reshape(D, H, W, C)
        return y * self.p[name + ".weight"] + self.p[name + ".bias"]

    def frequency(self, a, t):
        lin = lambda n, v: F.linear(v, self.p[a + n + ".weight"], self.p[a + n + ".bias"])
        g = lin("freq_mlp.4", F.gelu(lin("freq_mlp.2", F.gelu(lin("freq_mlp.0", t)))))
        h = F.gelu(lin("freq_lowrank.2", F.gelu(lin("freq_lowrank.0", t))))
        u, v = lin("freq_u", h), lin("freq_v", h)
        lead = t.shape[:-1]
        return torch.complex(g[..., 0], g[..., 1]), u.reshape(*lead, self.C, RANK), v.reshape(*lead, RANK, self.C)

    def gated(self, a, x):
        return x * torch.sigmoid(self.mlp(a + "input_gate", ".0.weight", ".2.weight", x))

    def weight(self, a):
        return torch.complex(self.p[a + "weight_real"], self.p[a + "weight_imag"])

    def plane(self, a, x):
        D, H, W, C = x.shape
        s = torch.fft.rfft2(self.gated(a, x), dim=(1, 2))
        ky = torch.fft.fftfreq(H, d=SPACING, dtype=torch.float64, device=x.device) * 1e5
        kx = torch.fft.rfftfreq(W, d=SPACING, dtype=torch.float64, device=x.device) * 1e5
        ky, kx = torch.meshgrid(ky, kx, indexing="ij")
        t = torch.stack([kx, ky, torch.sqrt(kx ** 2 + ky ** 2 + 1e-12), torch.sign(ky)], -1)
        g, u, v = self.frequency(a, t)
        low = torch.einsum("dhwi,hwri->dhwr", s, v.to(s.dtype))
        s = (s @ self.weight(a)) * g[..., None] + torch.einsum("dhwr,hwor->dhwo", low, u.to(s.dtype))
        return self.mlp(a + "post", ".0.weight", ".2.weight", torch.fft.irfft2(s, s=(H, W), dim=(1, 2)))

    def column(self, a, x):
        """The height operator: Filon integrals of the piecewise-linear column, mixing, the inverse sum."""
        c, p = self.c, self.p
        D, H, W, C = x.shape
        k = (2 * math.pi * torch.arange(c["modes"], dtype=torch.float32) / REFERENCE_LENGTH).double().to(x.device)
        each = c["columns"]
        z = self.low.permute(1, 2, 0) if each else self.low[:, 0, 0]          # [(H, W,) D]
        dz = (z[..., 1:] - z[..., :-1]).abs().median(-1).values[..., None]
        top = math.pi / dz
        keep = int((k < top.max()).sum())        # the taper is zero from the Nyquist wavenumber on
        k = k[:keep]
        taper = 0.5 * (1 + torch.cos(math.pi * ((k - 2 * top / 3) / (top / 3)).clamp(0, 1)))
        scale = taper * torch.where(torch.arange(keep, device=x.device) == 0, 1.0, 2.0).double() / REFERENCE_LENGTH
        near, far = z[..., :-1, None], z[..., 1:, None]
        h = (far - near).abs()
        th = h * k
        small = th < 1e-2
        t = torch.where(small, 1.0, th)
        cos, sin = torch.cos(t), torch.sin(t)
        up = torch.complex(torch.where(small, 0.5 - th ** 2 / 8, (cos + t * sin - 1) / t ** 2),
                           torch.where(small, -th / 3 + th ** 3 / 30, (t * cos - sin) / t ** 2))
        down = torch.complex(torch.where(small, 0.5 - th ** 2 / 24, sin / t - (cos + t * sin - 1) / t ** 2),
                             torch.where(small, -th / 6 + th ** 3 / 120, (cos - 1) / t - (t * cos - sin) / t ** 2))
        angle = torch.minimum(near, far) * k
        turn = torch.complex(h * torch.cos(angle), -h * torch.sin(angle))
        rising = near <= far
        q = F.pad(torch.where(rising, turn * down, turn * up), (0, 0, 0, 1)) \
            + F.pad(torch.where(rising, turn * up, turn * down), (0, 0, 1, 0))   # [(H, W,) D, M]
        xg = self.gated(a, x) + self.z[..., None] * p[a + "z_proj.weight"].reshape(C)
        into = "dhwc,hwdm->mhwc" if each else "dhwc,dm->mhwc"
        s = torch.complex(torch.einsum(into, xg, q.real), torch.einsum(into, xg, q.imag))
        f = k * FEATURE_WAVELENGTH / (2 * math.pi)
        f = f / (1 + f)
        g, u, v = self.frequency(a, torch.stack([f, f * f], -1))
        low = torch.einsum("mhwi,mri->mhwr", s, v.to(s.dtype))
        s = (s @ self.weight(a)) * g[:, None, None, None] + torch.einsum("mhwr,mor->mhwo", low, u.to(s.dtype))
        ph = z[..., None] * k
        back = "mhwc,hwdm->dhwc" if each else "mhwc,dm->dhwc"
        scale = scale[..., None, :]
        y = torch.einsum(back, s.real, torch.cos(ph) * scale) - torch.einsum(back, s.imag, torch.sin(ph) * scale)
        return self.mlp(a + "post", ".0.weight", ".2.weight", y)

    def block(self, i, x):
        p, a = self.p, "blocks.%d." % i
        s = F.gelu(self.norm(a + "norm_spec", self.plane(a + "spec.", x)))
        v = F.gelu(self.norm(a + "norm_vert", self.column(a + "vertical.", x)))
        gates = torch.sigmoid(self.mlp(a + "branch_gate", ".0.weight", ".2.weight", torch.cat([x, s, v], -1))
                              + p[a + "branch_gate.2.bias"])
        s, v = s * gates[..., :self.C], v * gates[..., self.C:]
        fused = self.mlp(a + "fuse", ".0.weight", ".2.weight", torch.cat([s, v], -1)) + 0.5 * (s + v)
        x = x + p[a + "res_fused"] * F.gelu(self.norm(a + "norm_fuse", fused))
        x = x + p[a + "res_pw"] * self.norm(a + "norm_pw", self.mlp(a + "pw", ".0.weight", ".2.weight", x))
        return x + p[a + "res_mlp"] * self.norm(a + "norm_mlp", self.mlp(a + "mlp.net", ".0.weight", ".3.weight", x))

    def head(self, x, x_in):
        p = self.p
        h = self.mlp("proj", "1.weight", "2.weight", x) + p["proj2.bias"]
        t, e, rho = (x_in[i] * p["std_X"][i] + p["mean_X"][i] for i in (0, 4, 5))
        kelvin, electrons = 10.0 ** t, 10.0 ** (e - 6.0)
        saha = math.log(0.5 * (_PLANCK / math.sqrt(2.0 * _PI * _MASS) / math.sqrt(_K)) ** 3) \
            + torch.log(electrons) - 1.5 * torch.log(kelvin)
        debye = 4.98e-4 * 5040.0 / kelvin * torch.sqrt(electrons * _K * kelvin)
        out, at = [], 0
        for atom in self.c["atoms"].split(","):
            weight, ion, ev, mass = _ATOMS[atom]
            # Debye multiples: 1, 3, 6, ... by stage, those up to the first level's stage counted from it
            count = [0, 0]
            for i in range(2, 21):
                count.append(count[-1] + i - 1)
            count = [n - count[ion[0]] if 1 <= i <= ion[0] else n for i, n in enumerate(count)]
            logits = torch.stack([h[..., at + i] + math.log(weight[i] / weight[0])
                                  - (_E / _K) / kelvin * (ev[i] - debye * count[ion[i]]) - (ion[i] - ion[0]) * saha
                                  for i in range(len(weight))])
            total = rho - torch.tensor(mass, dtype=torch.float32).item() + 6.0 * torch.tanh(h[..., at + len(weight)] / 6.0)
            out.append(total + torch.log_softmax(logits, 0) / math.log(10.0))
            at += len(weight) + 1
        return torch.cat(out)

    def __call__(self, x_in):
        x = x_in.permute(1, 2, 3, 0)
        x = F.gelu(self.norm("lift.1", x @ self.p["lift.0.weight"][:, :, 0, 0, 0].T))
        for i in range(self.c["layers"]):
            x = checkpoint(self.block, i, x, use_reentrant=False) if torch.is_grad_enabled() else self.block(i, x)
        return self.head(x, x_in)


def exact(case, seed):
    x, z, more = _inputs(case, seed)
    x, z = x[0].double(), z[0].double()
    if case["kind"] == "predict":
        with torch.no_grad():
            return _Exact(case, z)(x)[None].clone()
    if case["kind"] == "vjp":
        x.requires_grad_(True)
        z.requires_grad_(case["heights"])
        y = _Exact(case, z)(x)
        grads = torch.autograd.grad(y, (x, z) if case["heights"] else (x,), more[0].double())
        return [y.detach()[None], *(g[None] for g in grads)]
    import torch.autograd.forward_ad as forward_ad
    with torch.no_grad(), forward_ad.dual_level():
        y = _Exact(case, z)(forward_ad.make_dual(x, more[0].double()))
        return [v[None].clone() for v in forward_ad.unpack_dual(y)]
