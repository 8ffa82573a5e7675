"""Performance cases of the framework: the calls its users make, over the sizes, batches and types in use.

A case is a dict with a "kind" and its sizes. The kinds:
  adrt, adrt_T   the spatial transform and its transpose (adrtcore): exact integers and floating point
  inverse        FastHybridGpu / FastLpGpu .apply on device sinograms (whole reconstructions); in FP32 mode the images
                 go into the caller's FP32 buffer (out=), as they carry FP32 accuracy, in FP64 mode they are FP64
  cgls           pinv.cgls: a few iterations of the Moore-Penrose baseline (in finite precision a longer run depends on
                 the order of every sum, so its iterates cannot be compared)
  gram           gram.gram: R^T R of images through the offset frequencies (one packed pass each way)
  gram_freq      gram.gram_freq: the normal operator on frequency rows alone

The plans (spectral bounds, degrees, outer interval, dense operators) are kept per configuration by this module, as a
program that inverts more than one sinogram keeps its inverse object. Inputs come from plain torch code in this file,
so they do not depend on the framework's own kernels.
"""

import math

import numpy as np
import torch

import __graft_entry__ as entry

DTYPES = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64,
          "complex64": torch.complex64, "complex128": torch.complex128}
# inner degree cap p -> degree above which a row takes the exact dense filter, as the uneven workload pairs them
DENSE_CAPS = {8: None, 16: 12, 32: 16, 64: 16}
IMAGE_BUDGET = 64 * 256 * 256  # pixels of the largest batch
_handles = {}


def listed():
    return [
        # one small image at a time in the reference's own arithmetic: launches and latency
        {"name": "adrt f64 N=64 single", "kind": "adrt", "n": 6, "batch": 1, "dtype": "float64"},
        # a batch of 8-bit images as exact integers, both directions
        {"name": "adrt i32 N=256 b64", "kind": "adrt", "n": 8, "batch": 64, "dtype": "int32"},
        {"name": "adrt_T i32 N=256 b64", "kind": "adrt_T", "n": 8, "batch": 64, "dtype": "int32"},
        # a few large images, an odd batch
        {"name": "adrt_T f32 N=1024 b3", "kind": "adrt_T", "n": 10, "batch": 3, "dtype": "float32"},
        # the reference's call: one sinogram through L_p in FP64 (degree cap 16, every row polynomial)
        {"name": "lp f64 N=64 single", "kind": "inverse", "method": "lp", "n": 6, "batch": 1, "p": 16, "precision": "fp64"},
        # one sinogram at a time through the hybrid inverse (interactive use)
        {"name": "hybrid f32 N=256 single", "kind": "inverse", "method": "hybrid", "n": 8, "batch": 1, "p": 32,
         "precision": "fp32"},
        # the headline batch
        {"name": "hybrid f32 N=256 b64", "kind": "inverse", "method": "hybrid", "n": 8, "batch": 64, "p": 32,
         "precision": "fp32"},
        # one class of an uneven batch: an odd share of a small size, the other method
        {"name": "lp f32 N=128 b37", "kind": "inverse", "method": "lp", "n": 7, "batch": 37, "p": 16, "precision": "fp32"},
        # a small batch of a large size at a high degree (a serving lane)
        {"name": "hybrid f32 N=512 b6", "kind": "inverse", "method": "hybrid", "n": 9, "batch": 6, "p": 64,
         "precision": "fp32"},
        # the iterative baseline on a batch: the first iterations of a solve
        {"name": "cgls N=256 b16 x8", "kind": "cgls", "n": 8, "batch": 16, "iterations": 8},
        # the normal operator on images and on frequency rows alone
        {"name": "gram f32 N=256 b24", "kind": "gram", "n": 8, "batch": 24, "dtype": "float32"},
        {"name": "gram_freq c64 N=512 b9", "kind": "gram_freq", "n": 9, "batch": 9, "dtype": "complex64"},
    ]


def _batch(rng, n, most):
    """A batch size, spread over its logarithm, of at most `most` images and of the largest listed batch's pixels."""
    top = max(1, min(most, IMAGE_BUDGET >> (2 * n)))
    return max(1, min(top, int(round(math.exp(rng.uniform(0.0, math.log(top)))))))


def draw(rng):
    kind = rng.choice(["adrt", "adrt_T", "inverse", "inverse", "inverse", "cgls", "gram", "gram_freq"])
    if kind in ("adrt", "adrt_T"):
        n = rng.randint(5, 11)
        dtype = rng.choice(["int32", "int32", "float32", "float64", "int64"])
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 100), "dtype": dtype}
    if kind == "inverse":
        method = rng.choice(["lp", "hybrid"])
        if rng.random() < 0.15:
            n = rng.randint(5, 7)
            return {"kind": kind, "method": method, "n": n, "batch": _batch(rng, n, 8), "p": rng.choice([8, 16]),
                    "precision": "fp64"}
        n = rng.randint(5, 9)
        return {"kind": kind, "method": method, "n": n, "batch": _batch(rng, n, 64), "p": rng.choice([8, 16, 32, 64]),
                "precision": "fp32"}
    if kind == "cgls":
        n = rng.randint(6, 8)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 24), "iterations": rng.randint(5, 10)}
    if kind == "gram":
        n = rng.randint(5, 10)
        return {"kind": kind, "n": n, "batch": _batch(rng, n, 48), "dtype": rng.choice(["float32", "float32", "float64"])}
    n = rng.randint(5, 10)
    return {"kind": kind, "n": n, "batch": _batch(rng, n, 48), "dtype": rng.choice(["complex64", "complex64", "complex128"])}


# ---------------------------------------------------------------- the transform in plain torch (64 bits)
def _quadrants(x):
    """(B, N, N) -> (B, 4, N, N): the four quadrants' level-0 data, rows along the offset axis."""
    return torch.stack([x.flip(-1).transpose(-1, -2), x.flip(-2), x, x.flip(-1, -2).transpose(-1, -2)], 1)


def _unquadrants(s):
    """The transpose of _quadrants, summed over the quadrants."""
    return (s[:, 0].transpose(-1, -2).flip(-1) + s[:, 1].flip(-2)) + s[:, 2] + s[:, 3].transpose(-1, -2).flip(-1, -2)


def _shift_index(N, w, sign, device):
    """Row index h + sign (t + b) of every (h, t, b), into rows padded by w on the side that is left."""
    h = torch.arange(2 * N - 1, device=device)[:, None, None]
    t = torch.arange(w, device=device)[None, :, None]
    b = torch.arange(2, device=device)[None, None, :]
    return h + sign * (t + b) + (w if sign < 0 else 0)


def plain_adrt(n, x):
    """R x for x (B, N, N): (B, 4, 2N-1, N), rows h = -(N-1)..N-1."""
    N = 1 << n
    f = torch.nn.functional.pad(_quadrants(x), (0, 0, N - 1, 0))
    for m in range(1, n + 1):
        w = 1 << (m - 1)
        v = f.reshape(-1, 4, 2 * N - 1, N // (2 * w), 2, w)
        low = v[..., 0, :]
        high = torch.nn.functional.pad(v[..., 1, :], (0, 0, 0, 0, 0, w))
        out = torch.empty(v.shape[:4] + (w, 2), dtype=f.dtype, device=f.device)
        idx = _shift_index(N, w, 1, f.device)
        for b in range(2):
            i = idx[:, :, b][None, None, :, None, :].expand(low.shape)
            out[..., b] = low + torch.gather(high, 2, i)
        f = out.reshape(-1, 4, 2 * N - 1, N)
    return f


def plain_adrt_T(n, b):
    """R^T b for b (B, 4, 2N-1, N)."""
    N = 1 << n
    g = b
    h = torch.arange(2 * N - 1, device=b.device)[:, None] - (N - 1)
    for m in range(n, 0, -1):
        w = 1 << (m - 1)
        v = g.reshape(-1, 4, 2 * N - 1, N // (2 * w), w, 2)
        low = v[..., 0] + v[..., 1]
        idx = _shift_index(N, w, -1, b.device)
        high = torch.zeros_like(low)
        for c in range(2):
            i = idx[:, :, c][None, None, :, None, :].expand(low.shape)
            high = high + torch.gather(torch.nn.functional.pad(v[..., c], (0, 0, 0, 0, w, 0)), 2, i)
        inside = (h >= -torch.arange(w, device=b.device)[None, :]).to(b.dtype)[None, None, :, None, :]
        g = torch.stack([low * inside, high * inside], 4).reshape(-1, 4, 2 * N - 1, N)
    return _unquadrants(g[:, :, N - 1:, :])


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _phantoms(N, B, gen):
    """B images of ten random ellipses each (centres, semi-axes, angles and intensities as the repository's
    phantoms draw them), FP64 on the device."""
    u = torch.rand((6, 10, B, 1, 1), generator=gen, device="cuda", dtype=torch.float64)
    axis = torch.linspace(-1.0, 1.0, N, device="cuda", dtype=torch.float64)
    y, x = axis[None, :, None], axis[None, None, :]
    img = torch.zeros((B, N, N), device="cuda", dtype=torch.float64)
    for e in range(10):
        dx, dy = x - (1.2 * u[0, e] - 0.6), y - (1.2 * u[1, e] - 0.6)
        c, s = torch.cos(math.pi * u[4, e]), torch.sin(math.pi * u[4, e])
        r = ((dx * c + dy * s) / (0.05 + 0.35 * u[2, e])) ** 2 + ((dy * c - dx * s) / (0.05 + 0.35 * u[3, e])) ** 2
        img += (r <= 1.0) * (1.5 * u[5, e] - 0.5)
    return img


def _sinograms(n, B, gen):
    """Noisy sinograms of phantoms, sigma = 1e-3 max|b|, FP64."""
    b = plain_adrt(n, _phantoms(1 << n, B, gen))
    return b + 1e-3 * b.abs().amax(dim=(1, 2, 3), keepdim=True) * torch.randn(b.shape, generator=gen, device="cuda",
                                                                              dtype=torch.float64)


def _input(case, seed):
    gen = _generator(seed)
    n, B, N = case["n"], case["batch"], 1 << case["n"]
    kind = case["kind"]
    if kind in ("adrt", "adrt_T"):
        dtype = DTYPES[case["dtype"]]
        if dtype.is_floating_point:
            v = _phantoms(N, B, gen) if kind == "adrt" else _sinograms(n, B, gen)
        else:
            v = torch.randint(0, 256, (B, N, N), generator=gen, device="cuda")
            v = v if kind == "adrt" else plain_adrt(n, v)
        return v.to(dtype)
    if kind in ("inverse", "cgls"):
        return _sinograms(n, B, gen)
    if kind == "gram":
        return _phantoms(N, B, gen).to(DTYPES[case["dtype"]])
    shape = (B, 2 * N, N, 2)
    v = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    return torch.view_as_complex(v).to(DTYPES[case["dtype"]])


def _omega(case):
    real = torch.float32 if case["dtype"] == "complex64" else torch.float64
    w = 2 * np.pi * np.fft.fftfreq(2 << case["n"])
    return torch.from_numpy(w).to("cuda", real)


def _inverse(pkg, case):
    key = (case["method"], case["n"], case["p"], case["precision"])
    if key not in _handles:
        cls = pkg.FastHybridGpu if case["method"] == "hybrid" else pkg.FastLpGpu
        dense = DENSE_CAPS[case["p"]] if case["precision"] == "fp32" else None
        _handles[key] = cls(case["n"], deg_cap=case["p"], dense_cap=dense, precision=case["precision"])
    return _handles[key]


def prepare(case, seed):
    pkg = entry.load_package()
    kind = case["kind"]
    state = {"case": case, "in": _input(case, seed)}
    if kind in ("adrt", "adrt_T"):
        state["call"] = getattr(pkg.adrtcore, kind)
    elif kind == "inverse":
        state["inverse"] = _inverse(pkg, case)
        N = 1 << case["n"]
        if case["precision"] == "fp32":
            state["image"] = torch.empty((case["batch"], N, N), dtype=torch.float32, device="cuda")
    elif kind == "cgls":
        state["call"] = pkg.pinv.cgls
    elif kind == "gram":
        state["call"] = pkg.gram.gram
    else:
        state["call"], state["omega"] = pkg.gram.gram_freq, _omega(case)
    return state


def run(state):
    case, x = state["case"], state["in"]
    kind = case["kind"]
    if kind in ("adrt", "adrt_T"):
        return state["call"](case["n"], x, dtype=case["dtype"])
    if kind == "inverse":
        return state["inverse"].apply(x, out=state.get("image"))
    if kind == "cgls":
        images, history = state["call"](case["n"], x, tol=1e-30, maxit=case["iterations"])
        return [images, np.stack(history)]
    if kind == "gram":
        return state["call"](x)
    return state["call"](x, state["omega"])


def work(case):
    """Each input read once and each output written once; the operations of the transform's additions (N^2 per level,
    quadrant and image at least), and for the row operators 8N per butterfly level and row. An inverse counts the
    offset transforms and one pass of the row operators per outer iteration, with 20 iterations and a filter of degree
    4: less than any configuration here takes."""
    n, B, N = case["n"], case["batch"], 1 << case["n"]
    kind = case["kind"]
    image, sino = B * N * N, B * 4 * (2 * N - 1) * N
    if kind in ("adrt", "adrt_T"):
        return {"bytes": (image + sino) * DTYPES[case["dtype"]].itemsize, "flops": 4 * n * image}
    rows = B * 4 * N  # frequency rows of a packed pass
    fft = rows * 5 * N * (n + 1)
    if kind == "inverse":
        out = 4 if case["precision"] == "fp32" else 8
        return {"bytes": 8 * sino + out * image, "flops": 20 * (2 * fft + rows * 8 * N * 2 * n * 4)}
    if kind == "cgls":
        return {"bytes": 8 * (sino + image), "flops": case["iterations"] * (2 * 4 * n * image + 6 * sino + 6 * image)}
    if kind == "gram":
        return {"bytes": 2 * image * DTYPES[case["dtype"]].itemsize, "flops": 2 * fft + rows * 8 * N * 2 * n}
    size = 8 if case["dtype"] == "complex64" else 16
    return {"bytes": 2 * B * 2 * N * N * size, "flops": B * 2 * N * 8 * N * 2 * n}


# ---------------------------------------------------------------- the same results in 64 bits, plain torch
def _levels(Y, z, lo, hi):
    """B_hi ... B_lo on rows Y (..., K, N) at frequencies z (K,)."""
    N = Y.shape[-1]
    for m in range(lo, hi + 1):
        w = 1 << (m - 1)
        v = Y.reshape(Y.shape[:-1] + (N // (2 * w), 2, w))
        tw = z[:, None, None] ** torch.arange(w, device=Y.device, dtype=torch.float64)
        u = v[..., 1, :] * tw
        Y = torch.stack([v[..., 0, :] + u, v[..., 0, :] + u * z[:, None, None]], -1).reshape(Y.shape)
    return Y


def _levels_T(Y, z, lo, hi):
    N, zc = Y.shape[-1], z.conj()
    for m in range(hi, lo - 1, -1):
        w = 1 << (m - 1)
        v = Y.reshape(Y.shape[:-1] + (N // (2 * w), w, 2))
        tw = zc[:, None, None] ** torch.arange(w, device=Y.device, dtype=torch.float64)
        u = (v[..., 0] + v[..., 1] * zc[:, None, None]) * tw
        Y = torch.stack([v[..., 0] + v[..., 1], u], -2).reshape(Y.shape)
    return Y


class _Plain:
    """The explicit inverse of a case in FP64: x solves G x = y, which the fixed-degree outer iteration approximates to
    its tolerance of 1e-10. Spectral bounds by the 40 power steps from seeded starts, degrees, caps and the exact
    filter above the dense cap as the inverses define them; real strips, so frequencies 0..N."""

    def __init__(self, case):
        self.n, self.N, self.L = case["n"], 1 << case["n"], 2 << case["n"]
        n, N, L = self.n, self.N, self.L
        self.hybrid = case["method"] == "hybrid"
        self.lo = 2 if self.hybrid else 1
        tau, eps_in = 0.2 * N, 0.1
        k = torch.arange(L, device="cuda", dtype=torch.float64)
        z = torch.polar(torch.ones_like(k), 2 * math.pi * k / L)
        V = np.random.default_rng(0).standard_normal((L, N)) + 1j * np.random.default_rng(1).standard_normal((L, N))
        V = torch.from_numpy(V).to("cuda")
        for _ in range(40):
            V = self._gram(V, z)
            V = V / torch.linalg.vector_norm(V, dim=-1, keepdim=True)
        lam = 1.5 * (V.conj() * self._gram(V, z)).real.sum(-1)
        lam = torch.maximum(lam, lam[(-torch.arange(L, device="cuda")) % L]).clamp(min=1.0)[:N + 1]
        self.z, self.tau = z[:N + 1], tau
        root = torch.sqrt(1 + lam / tau)
        rate = ((root - 1) / (root + 1)).clamp(min=1e-12)
        deg = torch.ceil(math.log(eps_in / 2) / torch.log(rate)).clamp(min=2).clamp(max=case["p"])
        cap = DENSE_CAPS[case["p"]] if case["precision"] == "fp32" else None
        self.exact = deg > (cap if cap is not None else 1e9)
        self.deg = torch.where(self.exact, torch.ones_like(deg), deg)
        self.c, self.a = lam / (lam + 2 * tau), 2 / (lam + 2 * tau)
        if bool(self.exact.any()):
            ze = self.z[self.exact]
            eye = torch.eye(N, dtype=torch.complex128, device="cuda")[:, None, :].expand(N, len(ze), N)
            M = self._gram(eye, ze).permute(1, 2, 0)  # rows of the batch are images of unit vectors: columns of M
            self.F = torch.linalg.inv(M + tau * torch.eye(N, dtype=torch.complex128, device="cuda"))

    def _gram(self, Y, z):
        return _levels_T(_levels(Y, z, self.lo, self.n), z, self.lo, self.n)

    def _filter(self, y):
        """p_k(M) y per frequency (semi-iteration for (M + tau) z = y, d_k terms), or (M + tau)^{-1} y."""
        a, c, d = self.a[:, None], self.c[:, None], self.deg[:, None]
        z, zp, om = a * y, torch.zeros_like(y), torch.ones_like(c)
        for j in range(1, int(self.deg.max())):
            om = 1 / (1 - c * c / 2) if j == 1 else 1 / (1 - c * c * om / 4)
            on = (d > j).to(torch.float64)
            r = y - self._gram(z, self.z) - self.tau * z
            z, zp = z + on * (om * a * r + (om - 1) * (z - zp)), z
        if bool(self.exact.any()):
            z[..., self.exact, :] = torch.einsum("kij,...kj->...ki", self.F, y[..., self.exact, :])
        return z

    def _pass(self, strips, image):
        """One packed pass on strips (B, 4, L, N): row operators between the offset transforms, then the image."""
        Y, n = torch.fft.rfft(strips, dim=2), self.n
        if image:
            if self.hybrid:
                Y = _levels(Y, self.z, 1, 1)
            Y = self._gram(self._filter(Y), self.z)
        else:
            Y = self._filter(_levels_T(Y, self.z, self.lo, n))
        if self.hybrid:
            Y = _levels_T(Y, self.z, 1, 1)
        return _unquadrants(torch.fft.irfft(Y, n=self.L, dim=2)[:, :, :self.N])

    def G(self, x):
        return self._pass(torch.nn.functional.pad(_quadrants(x), (0, 0, 0, self.N)), True)

    def apply(self, b):
        N = self.N
        zero = torch.zeros_like(b[:, :, :1])
        y = self._pass(torch.cat([b[:, :, N - 1:], zero, b[:, :, :N - 1]], 2), False)
        x, r = torch.zeros_like(y), y.clone()
        p, rr = r.clone(), (y * y).sum((1, 2), keepdim=True)
        stop = 1e-25 * rr.max()
        for _ in range(400):  # conjugate gradients: G is symmetric positive definite
            if rr.max() <= stop:
                break
            q = self.G(p)
            alpha = rr / (p * q).sum((1, 2), keepdim=True).clamp(min=1e-300)
            x, r = x + alpha * p, r - alpha * q
            new = (r * r).sum((1, 2), keepdim=True)
            p, rr = r + (new / rr.clamp(min=1e-300)) * p, new
        return x


def _plain_cgls(n, b, iterations):
    """CGLS from zero; the history is ||R^T r||."""
    x = torch.zeros((b.shape[0], 1 << n, 1 << n), dtype=b.dtype, device=b.device)
    r, s = b.clone(), plain_adrt_T(n, b)
    p, gamma = s.clone(), (s * s).sum((1, 2))
    history = [torch.sqrt(gamma)]
    for _ in range(iterations):
        q = plain_adrt(n, p)
        alpha = gamma / (q * q).sum((1, 2, 3))
        x = x + alpha[:, None, None] * p
        r = r - alpha[:, None, None, None] * q
        s = plain_adrt_T(n, r)
        new = (s * s).sum((1, 2))
        p = s + (new / gamma)[:, None, None] * p
        gamma = new
        history.append(torch.sqrt(gamma))
    return [x, torch.stack(history, 1).cpu().numpy()]


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("adrt", "adrt_T") and case["dtype"].startswith("int"):
        return None  # whole numbers are compared as they are
    x = _input(case, seed)
    if kind in ("adrt", "adrt_T"):
        return (plain_adrt if kind == "adrt" else plain_adrt_T)(n, x.double())
    if kind == "inverse":
        return _Plain(case).apply(x)
    if kind == "cgls":
        return _plain_cgls(n, x, case["iterations"])
    if kind == "gram":
        x = x.double()
        out = torch.empty_like(x)
        for i in range(0, x.shape[0], 8):
            out[i:i + 8] = plain_adrt_T(n, plain_adrt(n, x[i:i + 8]))
        return out
    k = torch.arange(2 << n, device="cuda", dtype=torch.float64)
    z = torch.polar(torch.ones_like(k), _omega(case).double())
    Y = x.to(torch.complex128)
    return _levels_T(_levels(Y, z, 1, n), z, 1, n)
