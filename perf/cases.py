"""Performance cases: calls that programs make through motionest's public entry points.

A case is a dict of plain values.  `prepare` makes what such a program holds before the call
(inputs on the GPU from the seed alone, and the operator or problem that it keeps), `run` is one
call, `work` the bytes and operations that the call cannot do without, and `exact` its result in
complex128 by plain torch FFTs, without this package.

The inputs are the synthetic acquisitions that the package's own benchmark and tests use: an
ellipsoid phantom, Gaussian-bump coils of unit root-sum-of-squares, DISORDER masks, and rigid
motion of up to 3 degrees and 2 voxels per shot, with k-space made from them and noise added.
"""
import math

import numpy as np
import torch

from motionest.autograd import ForwardModel
from motionest.image_estimation import cg_solve
from motionest.joint_recon import JointRecon
from motionest.problem import SenseProblem, xyz_to_zxy
from motionest.sampling import disorder_masks
from motionest.simulation import coil_maps, generate_corrupted_kspace, phantom
from motionest.transform import RigidTransformCudaOptimzied, RigidTransformDerivativeCuda
from motionest.transform_estimation import LMState, lm_step
from motionest.utils import compute_transform_grids_voxel

AX3 = (-3, -2, -1)
NOISE = 1e-4  # std per real component, relative to the largest magnitude in k-space


def _case(name, op, shape, coils=0, shots=0, tile=(1, 1), accel=1, iters=0):
    return {"name": name, "op": op, "nx": shape[0], "ny": shape[1], "nz": shape[2],
            "coils": coils, "shots": shots, "tile_x": tile[0], "tile_y": tile[1],
            "accel": accel, "iters": iters}


def listed():
    return [
        # one rigid transform of a small image: launches and host work count most
        _case("transform_64", "transform", (64, 64, 48)),
        # its adjoint on a full-resolution image
        _case("adjoint_256", "adjoint", (256, 224, 176)),
        # one partial derivative on an acquisition matrix that is no power of two
        _case("partial_ragged", "partial", (180, 150, 126)),
        # one normal operator of CG-SENSE: the smallest workload, ...
        _case("normal_64", "normal", (64, 64, 48), 8, 16, (4, 4)),
        # ... the full-resolution one, ...
        _case("normal_256", "normal", (256, 224, 176), 32, 64, (16, 16), 2),
        # ... and an acquisition matrix with factors 3 and 5, tiles that divide it
        _case("normal_ragged", "normal", (160, 150, 126), 16, 20, (10, 10)),
        # a whole image step: the initial residual and the CG iterations at medium size
        _case("cg_128", "cg", (128, 112, 88), 16, 32, (8, 8), 2, 8),
        # a whole motion step over the full-resolution planes, on 32 readout points
        _case("lm_slab", "lm", (256, 224, 32), 32, 64, (16, 16), 2),
        # the same on a small matrix with factors 3, 5 and 7
        _case("lm_ragged", "lm", (90, 84, 70), 8, 12, (6, 6)),
        # the differentiable data term, forward and backward, for an image and its motion
        _case("grad_128", "grad", (128, 128, 96), 16, 32, (8, 8)),
        # the synthetic-data service: motion-corrupted k-space of one acquisition
        _case("simulate_128", "simulate", (128, 112, 88), 16, 32, (8, 8), 2),
        # a whole reconstruction from arrays: set-up, image and motion steps, objective
        _case("joint_64", "joint", (64, 64, 48), 8, 16, (4, 4), 1, 3),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _length(rng, lo, hi, multiple=1):
    """A line length between lo and hi, spread over the logarithm, a multiple of `multiple`
    that the package's FFTs take (prime factors up to 13)."""
    while True:
        n = multiple * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple))
        if lo <= n <= hi and _smooth(n):
            return n


def draw(rng):
    op = rng.choice(["transform", "adjoint", "partial", "normal", "normal", "cg", "lm", "grad",
                     "simulate", "joint"])
    if op in ("transform", "adjoint", "partial"):
        return _strip(_case("", op, tuple(_length(rng, 24, 256) for _ in range(3))))
    # coils x shots x voxels that a call may have (a motion step and a gradient move seven
    # volumes per shot, an image step several operators)
    most = {"normal": 2.0e9, "simulate": 1.0e9, "cg": 3.0e8, "lm": 2.0e8, "grad": 2.0e8,
            "joint": 5.0e7}[op]
    while True:
        tile = (rng.choice([2, 3, 4, 5, 6, 8, 10, 16]), rng.choice([2, 3, 4, 5, 6, 8, 10, 16]))
        X, Y = _length(rng, 32, 256, tile[0]), _length(rng, 32, 256, tile[1])
        Z = _length(rng, 12, 176)
        coils = rng.choice([4, 6, 8, 12, 16, 24, 32])
        shots = round(math.exp(rng.uniform(math.log(4), math.log(64))))
        accel = rng.choice([1, 2])
        per_shot = X * Y // accel // shots
        if coils * shots * X * Y * Z <= most and 16 <= per_shot <= 2000:
            break
    iters = {"cg": rng.randint(2, 8), "joint": rng.randint(1, 3)}.get(op, 0)
    return _strip(_case("", op, (X, Y, Z), coils, shots, tile, accel, iters))


def _strip(case):
    del case["name"]
    return case


# ------------------------------------------------------------- plain torch, any precision
# Volumes here are [Z, X, Y]; DIM[a] is the dimension of axis a (x, y, z).
DIM = (-2, -1, -3)
ROT_AXES = ((1, 2), (2, 0), (0, 1))  # the (tan, sin) shear axes of the rotations about x, y, z


class _Plain:
    """The rigid transform and the SENSE model by FFTs of whole volumes."""

    def __init__(self, shape, dtype):
        self.dtype = dtype
        self.k, r = [], []
        for a, n in enumerate(shape):
            view = [1, 1, 1]
            view[DIM[a]] = n
            for lo, hi, to in ((-n // 2, n // 2, r), (-np.pi, np.pi, self.k)):
                v = np.fft.fftshift(np.linspace(lo, hi, n, endpoint=False))
                to.append(torch.from_numpy(v).cuda().reshape(view))
        k = self.k
        self.tan = (r[2] * k[1], r[0] * k[2], r[1] * k[0])
        self.sin = (r[1] * k[2], r[2] * k[0], r[0] * k[1])

    def _along(self, v, f, a):
        f = f.to(self.dtype)
        return torch.fft.ifft(torch.fft.fft(v, dim=DIM[a]) * f, dim=DIM[a])

    def _factors(self, q, th, conj):
        s = -1.0 if conj else 1.0
        return (torch.exp(1j * s * math.tan(th / 2) * self.tan[q]),
                torch.exp(-1j * s * math.sin(th) * self.sin[q]))

    def rotate(self, v, q, th, conj=False):
        at, as_ = ROT_AXES[q]
        ft, fs = self._factors(q, th, conj)
        return self._along(self._along(self._along(v, ft, at), fs, as_), ft, at)

    def d_rotate(self, v, q, th):
        at, as_ = ROT_AXES[q]
        ft, fs = self._factors(q, th, False)
        dt = 1j * ((1 + math.tan(th / 2) ** 2) / 2) * self.tan[q] * ft
        ds = -1j * math.cos(th) * self.sin[q] * fs
        first = self._along(v, ft, at)
        mid = self._along(self._along(v, dt, at), fs, as_) + self._along(first, ds, as_)
        return self._along(mid, ft, at) + self._along(self._along(first, fs, as_), dt, at)

    def translate(self, v, p, conj=False, deriv=None):
        for a in range(3):
            f = torch.exp((1j if conj else -1j) * float(p[a]) * self.k[a])
            v = self._along(v, -1j * self.k[a] * f if a == deriv else f, a)
        return v

    def apply(self, v, p):
        for q in range(3):
            v = self.rotate(v, q, float(p[3 + q]))
        return self.translate(v, p)

    def adjoint(self, v, p):
        v = self.translate(v, p, conj=True)
        for q in (2, 1, 0):
            v = self.rotate(v, q, float(p[3 + q]), conj=True)
        return v

    def partial(self, v, p, i, order):
        for q in order:
            v = (self.d_rotate if i == 3 + q else self.rotate)(v, q, float(p[3 + q]))
        return self.translate(v, p, deriv=i if i < 3 else None)

    def samples(self, mps, mask, v):
        """M F_xy (mps v) of one shot: [C, Z, n] at the mask's points."""
        out = [torch.fft.fft2(mps[c:c + 8].to(self.dtype) * v, norm="ortho")[..., mask]
               for c in range(0, mps.shape[0], 8)]
        return torch.cat(out)

    def combine(self, mps, mask, K):
        """sum_c conj(mps_c) F_xy^H M^H K_c."""
        w = 0
        for c in range(0, mps.shape[0], 8):
            m = mps[c:c + 8].to(self.dtype)
            full = torch.zeros(m.shape, dtype=self.dtype, device=m.device)
            full[..., mask] = K[c:c + 8]
            w = w + (m.conj() * torch.fft.ifft2(full, norm="ortho")).sum(0)
        return w


def _to_xyz(v):
    return v.permute(1, 2, 0).contiguous()


# ------------------------------------------------------------------------------ inputs
def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _motion(case, seed):
    rng = np.random.default_rng(seed + 17)
    t = np.zeros((max(1, case["shots"]), 6))
    t[:, :3] = rng.uniform(-2, 2, (t.shape[0], 3))
    t[:, 3:] = np.deg2rad(rng.uniform(-3, 3, (t.shape[0], 3)))
    return t - t.mean(0) if t.shape[0] > 1 else t


def _volume(case, seed):
    """An uncentred [X, Y, Z] image with texture down to the voxel."""
    shape = _shape(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = phantom(shape, 10, seed, "cuda")
    n = torch.randn(shape + (2,), generator=g, device="cuda")
    return torch.fft.ifftshift(v + 0.05 * torch.view_as_complex(n)).contiguous()


def _acquisition(case, seed, with_kspace=True):
    """Centred masks [S, X, Y, 1] and uncentred everything else: image [X, Y, Z], maps
    [C, X, Y, Z], planes [S, X, Y], motion [S, 6], k-space [C, X, Y, Z]."""
    shape = _shape(case)
    a = {"x": _volume(case, seed), "t": _motion(case, seed)}
    a["mps"] = torch.fft.ifftshift(coil_maps(shape, case["coils"], seed, device="cuda"),
                                   dim=AX3).contiguous()
    a["masks"] = disorder_masks(shape[0], shape[1], (case["tile_x"], case["tile_y"]),
                                case["accel"], case["shots"])
    a["planes"] = np.fft.ifftshift(a["masks"][..., 0], axes=(-2, -1))
    if with_kspace:
        # [C, Z, X, Y] while it is made; points that two shots visit keep the later shot's value
        P = _Plain(shape, torch.complex64)
        m, x = a["mps"].permute(0, 3, 1, 2), xyz_to_zxy(a["x"])
        k = torch.zeros(m.shape, dtype=torch.complex64, device="cuda")
        for s in range(case["shots"]):
            mask = torch.from_numpy(a["planes"][s]).cuda()
            k[..., mask] = P.samples(m, mask, P.apply(x, a["t"][s]))
        k = torch.fft.fft(k, dim=-3, norm="ortho")
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        n = torch.randn(k.shape + (2,), generator=g, device="cuda")
        k = k + (NOISE * k.abs().max()) * torch.view_as_complex(n)
        a["ksp"] = k.permute(0, 2, 3, 1).contiguous()
        del k, n
    return a


def _start(a, seed):
    """What an iteration in mid-reconstruction holds: the image and motion, both still off."""
    rng = np.random.default_rng(seed + 5)
    off = rng.standard_normal(a["t"].shape) * np.array([0.3] * 3 + [0.006] * 3)
    return a["x"] * (1 - 0.1 * torch.rand(a["x"].shape, device="cuda",
                                          generator=torch.Generator(device="cuda")
                                          .manual_seed(seed + 2))), a["t"] + off


def prepare(case, seed):
    op, shape = case["op"], _shape(case)
    kg, rk = compute_transform_grids_voxel(shape, [1, 1, 1])
    s = {"op": op, "iters": case["iters"]}
    if op in ("transform", "adjoint"):
        s["T"] = RigidTransformCudaOptimzied(_motion(case, seed)[0], kg, rk)
        s["x"] = _volume(case, seed)
        return s
    if op == "partial":
        s["dT"] = RigidTransformDerivativeCuda(shape, _motion(case, seed)[0], kg, rk)
        s["x"] = _volume(case, seed)
        return s
    if op == "simulate":
        a = _acquisition(case, seed, with_kspace=False)
        s.update(x=torch.fft.fftshift(a["x"]), mps=torch.fft.fftshift(a["mps"], dim=AX3),
                 masks=a["masks"], t=a["t"])
        return s
    a = _acquisition(case, seed, with_kspace=op != "normal")
    if op == "joint":
        s.update(ksp=torch.fft.fftshift(a["ksp"], dim=AX3),
                 mps=torch.fft.fftshift(a["mps"], dim=AX3), masks=a["masks"], kg=kg, rk=rk)
        return s
    x, t = _start(a, seed)
    t = torch.from_numpy(t).cuda()
    if op == "grad":
        s["model"] = ForwardModel(a["ksp"], a["mps"], a["planes"][..., None], kg, rk)
        s["x"] = x.requires_grad_()
        s["theta"] = t.float().requires_grad_()
        return s
    s["pb"] = SenseProblem(a.get("ksp"), a["mps"], a["planes"], kg, rk, t)
    s["x"] = xyz_to_zxy(x)
    s["out"] = torch.empty_like(s["x"])
    if op == "lm":
        s.update(t=t, work=LMState(case["shots"], t.device))
    return s


def run(s):
    op = s["op"]
    if op == "transform":
        return s["T"].apply(s["x"])
    if op == "adjoint":
        return s["T"].adjoint(s["x"])
    if op == "partial":
        return s["dT"].apply(s["x"], 4)
    if op == "normal":
        return s["pb"].normal(s["x"], s["out"])
    if op == "cg":
        s["out"].copy_(s["x"])
        cg_solve(s["pb"], s["out"], s["iters"], 1e-6)
        return s["out"]
    if op == "lm":
        # the motion state is updated in place: each pass takes the step from the same start
        t = s["t"].clone()
        damp = torch.ones(t.shape[0], dtype=torch.float64, device=t.device)
        flags = torch.zeros(t.shape[0], dtype=torch.uint8, device=t.device)
        image = lm_step(s["pb"], s["x"], t, damp, flags, s["work"], out=s["out"])
        return {"image": image, "t": t.float(), "damp": damp.float()}
    if op == "grad":
        loss = s["model"].loss(s["x"], s["theta"])
        gx, gt = torch.autograd.grad(loss, (s["x"], s["theta"]))
        return {"x": gx, "theta": gt}
    if op == "simulate":
        return generate_corrupted_kspace(s["x"], s["mps"], s["masks"], s["t"])
    if op == "joint":
        app = JointRecon(s["ksp"], s["mps"], s["masks"], s["kg"], s["rk"], max_cg_iter=5,
                         max_joint_iter=s["iters"])
        x, t = app.run()
        return {"image": x, "t": t.float()}
    raise ValueError(op)


# -------------------------------------------------------------------------------- work
def work(case):
    X, Y, Z = _shape(case)
    V, C, S = X * Y * Z, case["coils"], case["shots"]
    lg = {"x": math.log2(X), "y": math.log2(Y), "z": math.log2(Z)}
    pair = {a: 10.0 * V * b + 6.0 * V for a, b in lg.items()}  # FFT, factor, inverse FFT
    # three shears per rotation (y z y, z x z, x y x) and the ramp along y; the ramps along x
    # and z ride in shears
    T = 3 * (pair["x"] + pair["y"] + pair["z"]) + pair["y"]
    rot = {0: 2 * pair["y"] + pair["z"], 1: 2 * pair["z"] + pair["x"], 2: 2 * pair["x"] + pair["y"]}
    op = case["op"]
    if op in ("transform", "adjoint"):
        return {"bytes": 16.0 * V, "flops": T}
    if op == "partial":
        return {"bytes": 16.0 * V, "flops": rot[0] + rot[2] + 2 * rot[1] +
                pair["x"] + pair["y"] + pair["z"]}
    per = X * Y // case["accel"] // S  # samples of a shot in one plane
    # SENSE model of one volume of one shot: map product, FFT along y, sums along x at the
    # samples; its adjoint costs the same
    fwd = C * (6.0 * V + 5.0 * V * lg["y"] + 8.0 * per * X * Z)
    maps, data = 8.0 * C * V, 8.0 * C * Z * per * S
    if op == "normal":
        return {"bytes": maps + 16.0 * V + 4.0 * per * S, "flops": S * (2 * T + 2 * fwd)}
    if op == "cg":
        return {"bytes": maps + data + 16.0 * V,
                "flops": (1 + case["iters"]) * S * (2 * T + 2 * fwd)}
    # T x and the six partials, sharing the rotations before the differentiated one
    jac = T + sum(rot.values()) + 9 * (pair["x"] + pair["y"] + pair["z"])
    if op == "lm":
        return {"bytes": maps + data + 16.0 * V, "flops": S * (jac + 7 * fwd + T + fwd) + T}
    if op == "grad":
        return {"bytes": maps + data + 24.0 * V,
                "flops": S * (T + fwd + jac + 2 * fwd + 2 * T + 2 * fwd)}
    zfft = 5.0 * C * V * lg["z"]
    if op == "simulate":
        return {"bytes": 2 * maps + 8.0 * V, "flops": S * (T + fwd) + zfft}
    step = 6 * S * (2 * T + 2 * fwd) + S * (jac + 7 * fwd + T + fwd) + T
    return {"bytes": 2 * maps + 8.0 * V, "flops": case["iters"] * step + 2 * zfft}


# ------------------------------------------------------------------------------- exact
def _data(a, P):
    """The shots' samples of the hybrid (IFFT_z) k-space: a list of [C, Z, n], and the masks."""
    kh = torch.fft.ifft(a["ksp"].permute(0, 3, 1, 2).to(P.dtype), dim=-3, norm="ortho")
    masks = [torch.from_numpy(p).cuda() for p in a["planes"]]
    return [kh[..., m].clone() for m in masks], masks


def _residual(P, m, y, masks, x, t):
    """sum_s T_s^H C^H F^H M_s (y_s - F C T_s x)."""
    out = torch.zeros_like(x)
    for s, mask in enumerate(masks):
        K = P.samples(m, mask, P.apply(x, t[s]))
        out = out + P.adjoint(P.combine(m, mask, y[s] - K), t[s])
    return out


def _normal(P, m, masks, x, t):
    out = torch.zeros_like(x)
    for s, mask in enumerate(masks):
        K = P.samples(m, mask, P.apply(x, t[s]))
        out = out + P.adjoint(P.combine(m, mask, K), t[s])
    return out


def _cg(P, m, y, masks, x, t, iters):
    rss = (m.to(P.dtype).abs() ** 2).sum(0)
    pre, sup = 1 / (rss + 1e-3), rss > 0.1
    r = sup * _residual(P, m, y, masks, x, t)
    z = pre * r
    p, rz = z, (r.conj() * z).sum().real
    for _ in range(iters):
        Ap = sup * _normal(P, m, masks, p, t)
        al = rz / (p.conj() * Ap).sum().real
        x, r = x + al * p, r - al * Ap
        z = pre * r
        new = (r.conj() * z).sum().real
        if math.sqrt(abs(float(new))) < 1e-6:
            break
        p, rz = z + (new / rz) * p, new
    return x


def _lm(P, m, y, masks, x, t, damp):
    """One damped Gauss-Newton step of every shot and the removal of the mean."""
    t, damp = t.copy(), damp.copy()
    for s, mask in enumerate(masks):
        r = P.samples(m, mask, P.apply(x, t[s])) - y[s]
        J = [P.samples(m, mask, P.partial(x, t[s], i, (2, 1, 0))) for i in range(6)]
        dot = lambda u, v: float((u.conj() * v).sum().real)  # noqa: E731
        g = np.array([dot(r, j) for j in J])
        H = np.array([[dot(u, v) for v in J] for u in J]) + damp[s] * np.eye(6)
        new = t[s] - np.linalg.solve(H, g)
        r1 = P.samples(m, mask, P.apply(x, new)) - y[s]
        if dot(r1, r1) < dot(r, r):
            t[s], damp[s] = new, max(damp[s] / 5, 1e-4)
        else:
            damp[s] = min(damp[s] * 1.5, 1e16)
    mean = t.mean(0)
    return P.apply(x, mean), t - mean, damp


def exact(case, seed):
    op, shape = case["op"], _shape(case)
    P = _Plain(shape, torch.complex128)
    if op in ("transform", "adjoint", "partial"):
        x, p = xyz_to_zxy(_volume(case, seed)).to(P.dtype), _motion(case, seed)[0]
        if op == "transform":
            return _to_xyz(P.apply(x, p))
        return _to_xyz(P.adjoint(x, p) if op == "adjoint" else P.partial(x, p, 4, (2, 1, 0)))
    volumes = {"normal": 1, "simulate": 1, "grad": 3, "lm": 8, "cg": 9, "joint": 40}[op]
    if case["coils"] * case["shots"] * shape[0] * shape[1] * shape[2] * volumes > 3.0e10:
        return None
    a = _acquisition(case, seed, with_kspace=op not in ("normal", "simulate"))
    m = a["mps"].permute(0, 3, 1, 2)
    if op == "simulate":
        k = torch.zeros(m.shape, dtype=P.dtype, device="cuda")
        x = xyz_to_zxy(a["x"]).to(P.dtype)
        for s in range(case["shots"]):
            mask = torch.from_numpy(a["planes"][s]).cuda()
            k[..., mask] += P.samples(m, mask, P.apply(x, a["t"][s]))
        k = torch.fft.fft(k, dim=-3, norm="ortho").permute(0, 2, 3, 1)
        return torch.fft.fftshift(k, dim=AX3)
    if op == "joint":
        y, masks = _data(a, P)
        full = torch.fft.ifftn(a["ksp"].to(P.dtype), dim=AX3, norm="ortho")
        top = full.abs().max()
        y = [v / top for v in y]
        x = torch.zeros((shape[2], shape[0], shape[1]), dtype=P.dtype, device="cuda")
        t, damp = np.zeros_like(a["t"]), np.ones(case["shots"])
        sup = (m.to(P.dtype).abs() ** 2).sum(0) > 0.1
        for _ in range(case["iters"]):
            x = _cg(P, m, y, masks, x, t, 5)
            x, t, damp = _lm(P, m, y, masks, x, t, damp)
            x = x * sup
        return {"image": torch.fft.fftshift(_to_xyz(x) * top), "t": torch.from_numpy(t)}
    x, t = _start(a, seed)
    x = xyz_to_zxy(x).to(P.dtype)
    if op == "normal":
        masks = [torch.from_numpy(p).cuda() for p in a["planes"]]
        sup = (m.to(P.dtype).abs() ** 2).sum(0) > 0.1
        return sup * _normal(P, m, masks, x, t)
    y, masks = _data(a, P)
    if op == "cg":
        return _cg(P, m, y, masks, x, t, case["iters"])
    if op == "lm":
        image, t, damp = _lm(P, m, y, masks, x, t, np.ones(case["shots"]))
        return {"image": image, "t": torch.from_numpy(t), "damp": torch.from_numpy(damp)}
    t = t.astype(np.float32).astype(np.float64)
    gx, gt = torch.zeros_like(x), np.zeros_like(t)
    for s, mask in enumerate(masks):
        r = P.samples(m, mask, P.apply(x, t[s])) - y[s]
        w = P.combine(m, mask, r)
        gx += P.adjoint(w, t[s])
        for i in range(6):
            gt[s, i] = float((w.conj() * P.partial(x, t[s], i, (0, 1, 2))).sum().real)
    return {"x": _to_xyz(gx), "theta": torch.from_numpy(gt)}
