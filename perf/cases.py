"""The work a user of this engine has it do, as cases that can be timed and compared.

Each kind is one public entry point:

* ``session``: ``SSB.from_array(counts).reconstruct(...)``, one acquisition in
  HBM to an object wave (with the default loss or without), the scan padded by
  the engine's rule. Interactive use and small scans.
* ``stream``: ``ColdReconstructor.run()``, acquisitions of one shape arriving
  one after the other (a detector feeding scans). The production path.
* ``score``: ``variance_loss_batch`` of a prepared dataset, what fits, sweeps
  and the learned proposal's refinement spend their time in.
* ``terms``: ``variance_loss_batch_full``, the same with the 14-term chi.
* ``train``: one step of the proposer's MLP, forward, backward and Adam.
* ``decode`` / ``encode``: bitshuffle + LZ4 chunks to u16 frames and back.
* ``join``: the drift-corrected complex mean of a time series of object waves.

Counts are Poisson draws from the package's synthetic acquisition (300 kV, a
weak-phase atom lattice, soft aperture), laid out from a 64 x 64-position tile
of expected intensities so that large scans are made quickly.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from quantem.gpu_b200 import SSB, B200SSBBackend
from quantem.gpu_b200 import decode as qdecode
from quantem.gpu_b200 import temporal
from quantem.gpu_b200.physics import wavelength_angstrom
from quantem.gpu_b200.pipeline import ColdReconstructor
from quantem.gpu_b200.proposer import MLP, Proposer
from quantem.gpu_b200.synthetic import SyntheticSpec, draw_aberrations, generate

VOLTAGE_KV = 300.0
STEP_A = 0.5
TILE = 64
BASE_DOSE = 4.0e5  # expected counts of the tile, rounded to integers
FULL_NM = ((1, 0), (1, 2), (2, 1), (2, 3), (3, 0), (3, 2), (3, 4),
           (4, 1), (4, 3), (4, 5), (5, 0), (5, 2), (5, 4), (5, 6))


def listed():
    return [
        # the smallest acquisition of the tests, one reconstruction with its
        # diagnostic loss: launches, synchronisations and padding count
        {"name": "session_32x32_det64", "kind": "session", "rows": 32, "cols": 32, "det": 64,
         "radius": 12.0, "semi": 20.0, "dose": 1000.0, "rotation": 0.0, "loss": True, "bits": 16},
        # an uneven scan (the sweep's third), padded to 256 x 256
        {"name": "session_160x120_det128", "kind": "session", "rows": 160, "cols": 120, "det": 128,
         "radius": 24.0, "semi": 20.0, "dose": 1000.0, "rotation": 12.0, "loss": True, "bits": 16},
        # the headline: 128 x 128 scan, 128 x 128 detector, u16 in HBM to phase
        {"name": "stream_128x128_det128", "kind": "stream", "n": 128, "det": 128,
         "radius": 24.0, "semi": 20.0, "dose": 1000.0},
        # a large acquisition: 8.6 GB, about 4000 BF pixels
        {"name": "stream_512x512_det128", "kind": "stream", "n": 512, "det": 128,
         "radius": 36.0, "semi": 25.0, "dose": 1000.0},
        # one batch of a plain sweep on the headline dataset
        {"name": "score_128_64c", "kind": "score", "rows": 128, "cols": 128, "det": 128,
         "radius": 24.0, "semi": 20.0, "n_cand": 64, "c30": False},
        # one round of the proposal's refinement on a 64 x 64 scan
        {"name": "score_64_8c_c30", "kind": "score", "rows": 64, "cols": 64, "det": 64,
         "radius": 12.0, "semi": 20.0, "n_cand": 8, "c30": True},
        # part of a sweep on a 256 x 256 scan
        {"name": "score_256_16c_c30", "kind": "score", "rows": 256, "cols": 256, "det": 128,
         "radius": 24.0, "semi": 20.0, "n_cand": 16, "c30": True},
        # a batch of higher-order candidates
        {"name": "terms_128_8c", "kind": "terms", "rows": 128, "cols": 128, "det": 128,
         "radius": 24.0, "semi": 20.0, "n_cand": 8},
        # one training step at the proposer's batch size
        {"name": "train_256", "kind": "train", "batch": 256},
        # a stored 128 x 128 acquisition decoded, and a smaller one written
        {"name": "decode_16384_det128", "kind": "decode", "frames": 16384, "det": 128,
         "radius": 24.0, "semi": 20.0, "dose": 1000.0},
        {"name": "encode_4096_det128", "kind": "encode", "frames": 4096, "det": 128,
         "radius": 24.0, "semi": 20.0, "dose": 1000.0},
        # a time series of reconstructions of the headline size
        {"name": "join_256x128x128", "kind": "join", "frames": 256, "rows": 128, "cols": 128,
         "reference": True, "aligned": False},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["session", "stream", "score", "terms", "train", "decode", "encode", "join"])
    det = rng.randint(48, 160)
    optics = {"det": det, "radius": round(det * rng.uniform(0.15, 0.25), 2), "semi": 20.0}
    dose = round(math.exp(rng.uniform(math.log(50.0), math.log(20000.0))), 1)
    if kind == "session":
        return {"kind": kind, "rows": log_int(24, 256), "cols": log_int(24, 256), **optics,
                "dose": dose, "rotation": round(rng.uniform(-90.0, 90.0), 2),
                "loss": rng.random() < 0.5, "bits": rng.choice([8, 16, 16])}
    if kind == "stream":
        n = rng.choice([128, 256, 512])
        if n == 512 and det > 128:
            optics = {"det": 128, "radius": round(optics["radius"] * 128 / det, 2), "semi": 20.0}
        return {"kind": kind, "n": n, **optics, "dose": dose}
    if kind == "score":
        n = rng.choice([64, 96, 128, 192, 256, 512])
        most = {64: 64, 96: 64, 128: 64, 192: 24, 256: 24, 512: 2}[n]
        return {"kind": kind, "rows": n, "cols": n - rng.randint(0, n // 3), **optics,
                "n_cand": log_int(1, most), "c30": rng.random() < 0.5}
    if kind == "terms":
        n = rng.choice([64, 128, 128, 256])
        return {"kind": kind, "rows": n, "cols": n - rng.randint(0, n // 4), **optics,
                "n_cand": log_int(1, 2 if n == 256 else 8)}
    if kind == "train":
        return {"kind": kind, "batch": 16 * rng.randint(4, 32)}
    if kind in ("decode", "encode"):
        det = rng.randint(48, 192)
        frames = min(log_int(256, 16384 if kind == "decode" else 8192), (1 << 28) // (det * det))
        return {"kind": kind, "frames": frames, "det": det,
                "radius": round(det * rng.uniform(0.15, 0.25), 2), "semi": 20.0, "dose": dose}
    rows, cols = rng.choice([64, 128, 256, 512]), rng.choice([64, 128, 256, 512])
    frames = min(log_int(8, 300), (1 << 24) // (rows * cols))
    return {"kind": kind, "frames": frames, "rows": rows, "cols": cols,
            "reference": rng.random() < 0.7, "aligned": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _counts(rows, cols, case, dose, seed, bits=16):
    """uint counts [rows, cols, det, det] on the GPU, and the aberrations they were made with."""
    det = case["det"]
    ab = draw_aberrations(np.random.default_rng(seed), 1)[0]
    c10, c12, phi12 = (float(ab[0]) * 0.4, float(ab[1]) * 0.5, float(ab[2]))
    spec = SyntheticSpec(scan_shape=(min(rows, TILE), min(cols, TILE)), detector_shape=(det, det),
                         voltage_kV=VOLTAGE_KV, semiangle_mrad=case["semi"], scan_step_A=STEP_A,
                         det_sampling_mrad=case["semi"] / case["radius"], dose=BASE_DOSE,
                         C10=c10, C12=c12, phi12=phi12, seed=seed, poisson=False)
    base = generate(spec, device="cuda").counts.to(torch.int32).to(torch.float32) * (dose / BASE_DOSE)
    g = _generator(seed + 17)
    top = (1 << bits) - 1
    out = torch.empty((rows, cols, det, det), device="cuda",
                      dtype=torch.uint16 if bits == 16 else torch.uint8)
    for r in range(0, rows, TILE):
        for c in range(0, cols, TILE):
            tile = base[: min(TILE, rows - r), : min(TILE, cols - c)]
            draws = torch.poisson(tile, generator=g).clamp_(max=top)
            out[r:r + tile.shape[0], c:c + tile.shape[1]] = draws.to(torch.int32).to(out.dtype)
    return out, {"C10": c10, "C12": c12, "phi12": phi12}


def _candidates(case, seed):
    """[n_cand, 4] (C10, C12, phi12, C30) of the sweep ranges."""
    c = draw_aberrations(np.random.default_rng(seed + 5), case["n_cand"])
    if not case["c30"]:
        c[:, 3] = 0.0
    return c


def _terms(case, seed):
    """([n_cand, 14] magnitudes, [n_cand, 14] angles): 0.2 .. 4 rad of chi per
    term at the aperture edge, some terms off."""
    rng = np.random.default_rng(seed + 6)
    n = case["n_cand"]
    lam, alpha = wavelength_angstrom(VOLTAGE_KV), case["semi"] * 1e-3
    mags = np.empty((n, 14))
    angs = np.zeros((n, 14))
    for i, (order, m) in enumerate(FULL_NM):
        edge = rng.uniform(0.2, 4.0, n) * rng.choice([-1.0, 1.0], n) * (rng.random(n) < 0.8)
        mags[:, i] = edge * (order + 1) * lam / (2 * math.pi * alpha ** (order + 1))
        if m:
            mags[:, i] = np.abs(mags[:, i])
            angs[:, i] = rng.uniform(0, 2 * math.pi / m, n)
    return mags.astype(np.float32), angs.astype(np.float32)


def _waves(case, seed):
    """A time series of one object wave: drift, a global phase per frame, noise."""
    t, r, c = case["frames"], case["rows"], case["cols"]
    rng = np.random.default_rng(seed)
    shifts = rng.uniform(-3.0, 3.0, (t, 2)).astype(np.float32)
    theta = torch.as_tensor(rng.uniform(-math.pi, math.pi, t), device="cuda", dtype=torch.float32)
    g = _generator(seed)
    phase = 0.3 * torch.randn((r, c), device="cuda", generator=g)
    amp = 1.0 + 0.05 * torch.randn((r, c), device="cuda", generator=g)
    stack = torch.polar(amp, phase)[None] * torch.polar(torch.ones_like(theta), theta)[:, None, None]
    stack = stack + torch.complex(*(0.05 * torch.randn((t, r, c), device="cuda", generator=g)
                                    for _ in range(2)))
    return stack.contiguous(), torch.from_numpy(shifts)


def _backend(counts, case):
    return B200SSBBackend(counts, semiangle=case["semi"], scan_sampling=STEP_A,
                          det_sampling=case["semi"] / case["radius"], voltage_kV=VOLTAGE_KV)


def _side(case):
    """The scan size after padding."""
    longest = max(case["rows"], case["cols"])
    return next(s for s in (128, 256, 512, 1024) if longest <= s)


def _gradients(w, b, x, t):
    """Outputs, loss and gradients of the heads' winner-takes-all loss in 64 bits, in plain torch."""
    w, b = [v.double() for v in w], [v.double() for v in b]
    leaves = [v.detach().requires_grad_() for v in w + b]
    a = x.double()
    for i in range(4):
        a = a @ leaves[i] + leaves[4 + i]
        if i < 3:
            a = 0.5 * a * (1.0 + torch.erf(a / math.sqrt(2.0)))
    rows = torch.arange(len(x), device="cuda")
    weight = torch.tensor([1.0, 1.0, 1.0, 0.1], device="cuda", dtype=torch.float64)
    d = a.reshape(len(x), 4, 4) - t.double()[:, None]
    win = (d[..., :3] ** 2).sum(-1).argmin(1)
    share = torch.full(d.shape[:2], 0.05 / 3, device="cuda", dtype=torch.float64)
    share[rows, win] = 0.95
    each = (d * d * weight).sum(-1)
    grads = torch.autograd.grad((each * share).sum() / (len(x) * 4), leaves)
    return a.detach(), (each[rows, win].sum() / (len(x) * 4)).detach(), list(grads)


STEPS_TAKEN = 20


def _train_state(case, seed):
    """The network with an optimiser some steps in (moments of two other
    batches' gradients), and a batch of forward-model features."""
    m = case["batch"]
    x, t, _ = Proposer("cuda", seed=seed).make_data(3 * m, seed)
    mlp = MLP("cuda", seed=seed)
    one, two = (_gradients(mlp.w_bf, mlp.b, x[k * m:(k + 1) * m], t[k * m:(k + 1) * m])[2]
                for k in (1, 2))
    for k, (g1, g2) in enumerate(zip(one, two)):
        mlp.m[k].copy_(0.5 * (g1 + g2))
        mlp.v[k].copy_(0.5 * (g1 * g1 + g2 * g2))
    mlp.t = STEPS_TAKEN
    return mlp, x[:m].contiguous(), t[:m].contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "session":
        counts, ab = _counts(case["rows"], case["cols"], case, case["dose"], seed, case["bits"])
        return {"case": case, "counts": counts, "ab": ab}
    if kind == "stream":
        counts, ab = _counts(case["n"], case["n"], case, case["dose"], seed)
        return {"case": case, "cold": ColdReconstructor(
            counts, semiangle=case["semi"], scan_sampling=STEP_A,
            det_sampling=case["semi"] / case["radius"], voltage_kV=VOLTAGE_KV,
            aberrations=(ab["C10"], ab["C12"], ab["phi12"], 0.0))}
    if kind in ("score", "terms"):
        counts, _ = _counts(case["rows"], case["cols"], case, 1000.0, seed)
        be = _backend(counts, case)
        cands = _candidates(case, seed) if kind == "score" else _terms(case, seed)
        return {"case": case, "be": be, "cands": cands}
    if kind == "train":
        mlp, x, t = _train_state(case, seed)
        return {"case": case, "mlp": mlp, "x": x, "t": t}
    if kind in ("decode", "encode"):
        frames = _frames(case, seed)
        if kind == "encode":
            # a file buffer that the packed chunks go to
            return {"case": case, "frames": frames,
                    "file": torch.zeros(frames.numel() + 4096, dtype=torch.uint8, device="cuda")}
        comp, offsets = qdecode.encode_bslz4(frames)
        return {"case": case, "comp": comp, "offsets": offsets}
    stack, shifts = _waves(case, seed)
    return {"case": case, "stack": stack, "shifts": shifts}


def _frames(case, seed):
    cols = -(-case["frames"] // TILE)
    counts, _ = _counts(TILE, cols, case, case["dose"], seed)
    return counts.reshape(-1, case["det"], case["det"])[:case["frames"]].contiguous()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "session":
        with SSB.from_array(state["counts"], voltage_kV=VOLTAGE_KV, semiangle_mrad=case["semi"],
                            scan_sampling_A=STEP_A, det_sampling=case["semi"] / case["radius"],
                            rotation_angle_deg=case["rotation"]) as ssb:
            result = ssb.reconstruct(state["ab"], compute_loss=case["loss"])
        if result.loss is None:
            return {"object": result.object_wave}
        return {"object": result.object_wave, "loss": result.loss}
    if kind == "stream":
        return {"phase": state["cold"].run()}
    if kind == "score":
        c = state["cands"]
        if case["n_cand"] == 1 and not case["c30"]:
            phase, loss = state["be"].reconstruct_with_loss(*(float(v) for v in c[0, :3]))
            return {"phase": phase, "loss": loss}
        return {"loss": state["be"].variance_loss_batch(c[:, 0], c[:, 1], c[:, 2],
                                                        c[:, 3] if case["c30"] else None)}
    if kind == "terms":
        return {"loss": state["be"].variance_loss_batch_full(*state["cands"])}
    if kind == "train":
        mlp = state["mlp"]
        out = mlp.forward(state["x"])
        loss = mlp.backward_and_step(state["t"], 1e-3)
        # the first moments carry the step's gradients
        return {"out": out, "loss": loss, "w": mlp.w, "b": mlp.b, "m": mlp.m}
    if kind == "decode":
        frames = qdecode.decode_bslz4(state["comp"], state["offsets"], (case["det"], case["det"]))
        return frames.view(torch.int16)  # the same bits, in a type that torch can index
    if kind == "encode":
        packed, offsets = qdecode.encode_bslz4(state["frames"])
        state["file"][:packed.numel()].copy_(packed)
        return {"file": state["file"], "bytes": packed.numel(), "offsets": offsets}
    got = temporal.join_object_waves(state["stack"], state["shifts"],
                                     phase_reference="first" if case["reference"] else "none",
                                     return_aligned_stack=case["aligned"])
    if case["aligned"]:
        return {"joined": got[0].object_wave, "aligned": got[1]}
    return {"joined": got.object_wave}


# ------------------------------------------------------------------- costs
def work(case):
    kind = case["kind"]
    if kind in ("session", "stream"):
        rows = case["n"] if kind == "stream" else case["rows"]
        cols = case["n"] if kind == "stream" else case["cols"]
        n = rows if kind == "stream" else _side(case)
        n_bf = math.pi * case["radius"] ** 2
        # a real 2D FFT and the Fourier sum over half the frequencies per BF pixel
        flops = n_bf * n * n * (2.5 * math.log2(n * n) + 30.0)
        if case.get("loss"):
            flops += n_bf * n * n * (2.5 * math.log2(n * n) + 40.0)
        return {"bytes": rows * cols * case["det"] ** 2 * (case.get("bits", 16) // 8) + 8 * n * n,
                "flops": flops}
    if kind in ("score", "terms"):
        n = _side(case)
        n_bf = math.pi * case["radius"] ** 2
        per = (2.5 * math.log2(n * n) + 40.0) if kind == "score" else (5.0 * math.log2(n * n) + 100.0)
        return {"bytes": 8 * n_bf * n * (n // 2 + 1) + 20 * case["n_cand"],
                "flops": case["n_cand"] * n_bf * n * n * per}
    if kind == "train":
        dims = (16384, 512, 512, 512, 16)
        params = sum(a * b + b for a, b in zip(dims, dims[1:]))
        m = case["batch"]
        # x read; master weights and both moments read and written, the BF16 copy
        # read and written
        return {"bytes": 2 * m * dims[0] + params * (24 + 4),
                "flops": m * (6.0 * params - 2.0 * dims[0] * dims[1])}
    if kind in ("decode", "encode"):
        return {"bytes": 2 * case["frames"] * case["det"] ** 2, "flops": 0}
    t, n = case["frames"], case["rows"] * case["cols"]
    return {"bytes": 8 * n * (t + 1 + (t if case["aligned"] else 0)),
            "flops": t * n * (10.0 * math.log2(n) + 20.0)}


def tolerance(case):
    """About four times what each path was measured to be off in 64 bits (the
    worst seen: object 7e-6 where aperture pairs nearly tie, losses 2e-7 and
    7e-7 with their fold, updated biases 1e-3 from BF16 activations)."""
    kind = case["kind"]
    if kind in ("session", "stream") or (kind == "score" and case["n_cand"] == 1):
        return {"rel": 3e-5}
    if kind == "score":
        return {"rel": 2e-6}
    if kind == "terms":
        return {"rel": 4e-6}
    if kind == "train":
        return {"rel": 4e-3, "max": 0.3}
    if kind in ("decode", "encode"):
        return "exact"
    return {"rel": 2e-6}


# ------------------------------------------------------- the same in 64 bits
def _pad(counts):
    """[rows, cols, K, K] int64 padded with the floored mean pattern to the square native size."""
    rows, cols = counts.shape[:2]
    n = next(s for s in (128, 256, 512, 1024) if max(rows, cols) <= s)
    if rows == cols == n:
        return counts
    fill = (counts.sum(dim=(0, 1)).double() / (rows * cols)).floor().to(counts.dtype)
    out = fill.expand(n, n, *fill.shape).contiguous()
    top, left = (n - rows) // 2, (n - cols) // 2
    out[top:top + rows, left:left + cols] = counts
    return out


class _Exact:
    """The reconstruction in 64 bits: BF selection (whose comparisons are made
    in float32), scan spectra, the corrected spectra per chunk of BF pixels."""

    def __init__(self, counts, case, rotation_deg=0.0):
        counts = counts if counts.dtype == torch.uint8 else counts.view(torch.int16)
        rows, cols, k = counts.shape[0], counts.shape[1], case["det"]
        n = next(s for s in (128, 256, 512, 1024) if max(rows, cols) <= s)
        if not rows == cols == n:
            wide = counts.to(torch.int32) & 0xFFFF
            counts = _pad(wide.long()).to(torch.int32).to(torch.int16)
        sums = torch.zeros((k, k), dtype=torch.int64, device="cuda")
        for r in range(n):
            sums += (counts[r].to(torch.int32) & 0xFFFF).sum(dim=0, dtype=torch.int64)
        mean = sums.cpu().numpy().astype(np.float32) / np.float32(n * n)
        wide = mean.astype(np.float64)
        probe = mean > np.float32(wide.mean()) + np.float32(wide.std())
        total = int(probe.sum())
        pr, pc = np.nonzero(probe)
        center = (float(np.float32(pr.sum()) / np.float32(total)),
                  float(np.float32(pc.sum()) / np.float32(total)))
        br, bc = np.nonzero(mean > 0)
        d2 = ((br.astype(np.float32) - np.float32(center[0])) ** 2
              + (bc.astype(np.float32) - np.float32(center[1])) ** 2)
        keep = d2 <= np.float32(total / math.pi)
        br, bc = br[keep], bc[keep]
        self.n, self.lam = n, wavelength_angstrom(VOLTAGE_KV)
        self.semi, self.pitch = case["semi"] * 1e-3, case["semi"] / case["radius"] * 1e-3
        dk = self.pitch / self.lam
        th = -math.radians(rotation_deg)
        kr, kc = (br - center[0]) * dk, (bc - center[1]) * dk
        self.kx = torch.as_tensor(kr * math.cos(th) + kc * math.sin(th), device="cuda")
        self.ky = torch.as_tensor(-kr * math.sin(th) + kc * math.cos(th), device="cuda")
        self.counts, self.lin = counts.reshape(n * n, k * k), torch.as_tensor(br * k + bc, device="cuda")
        self.dc = float(sums.reshape(-1)[self.lin].double().mean())
        self.q = torch.fft.fftfreq(n, STEP_A, dtype=torch.float64, device="cuda")
        self.n_bf = int(self.lin.numel())
        self.chunk = max(1, (1 << 22) // (n * n))

    def spectra(self, s):
        cols = self.counts[:, self.lin[s:s + self.chunk]].to(torch.int32) & 0xFFFF
        return torch.fft.fft2(cols.T.reshape(-1, self.n, self.n).double())

    def _probe(self, dx, dy, ab):
        r2 = dx * dx + dy * dy
        edge = ((self.semi - self.lam * r2.sqrt()) / self.pitch + 0.5).clamp_(0.0, 1.0)
        if len(ab) == 4:
            c10, c12, phi, c30 = ab
            f = math.pi * self.lam
            chi = f * (c10 * r2 + c12 * ((dx * dx - dy * dy) * math.cos(2 * phi)
                                         + 2 * dx * dy * math.sin(2 * phi)))
            if c30:
                chi = chi + 0.5 * f * self.lam ** 2 * c30 * r2 * r2
        else:
            alpha, ang = self.lam * r2.sqrt(), torch.atan2(dy, dx)
            chi = torch.zeros_like(alpha)
            for (order, m), mag, a in zip(FULL_NM, ab[:14], ab[14:]):
                if mag:
                    chi += (2 * math.pi / self.lam * mag / (order + 1)) * alpha ** (order + 1) \
                        * torch.cos(m * (ang - a))
        return torch.polar(edge, -chi)

    def corrected(self, s, g, ab):
        kx, ky = (v[s:s + self.chunk, None, None] for v in (self.kx, self.ky))
        qx, qy = self.q[None, :, None], self.q[None, None, :]
        pk = self._probe(kx, ky, ab)
        gamma = self._probe(qx - kx, qy - ky, ab) * pk.conj()
        gamma -= self._probe(qx + kx, qy + ky, ab).conj() * pk
        c = g * gamma.conj() / gamma.abs().clamp_(min=1e-8)
        c[:, 0, 0] = self.dc
        return c

    def object(self, ab):
        total = 0
        for s in range(0, self.n_bf, self.chunk):
            total = total + self.corrected(s, self.spectra(s), ab).sum(dim=0)
        return torch.fft.ifft2(total / self.n_bf)

    def losses(self, abs_):
        s1 = [0.0] * len(abs_)
        s2 = [0.0] * len(abs_)
        for s in range(0, self.n_bf, self.chunk):
            g = self.spectra(s)
            for i, ab in enumerate(abs_):
                ang = torch.fft.ifft2(self.corrected(s, g, ab)).angle()
                s1[i] = s1[i] + ang.sum(dim=0)
                s2[i] = s2[i] + (ang * ang).sum()
        means = [v / self.n_bf for v in s1]
        loss = [(q / (self.n_bf * self.n ** 2) - (m * m).mean()) for q, m in zip(s2, means)]
        return torch.stack(loss), means


def _train_exact(case, seed):
    mlp, x, t = _train_state(case, seed)
    out, loss, grads = _gradients(mlp.w_bf, mlp.b, x, t)
    c1, c2 = 1.0 - 0.9 ** (STEPS_TAKEN + 1), 1.0 - 0.999 ** (STEPS_TAKEN + 1)
    new, moments = [], []
    for i, (p, m, v, g) in enumerate(zip(mlp.w + mlp.b, mlp.m, mlp.v, grads)):
        p = p.double()
        m = 0.9 * m.double() + 0.1 * g
        v = 0.999 * v.double() + 0.001 * g * g
        new.append(p - 1e-3 * ((m / c1) / ((v / c2).sqrt() + 1e-8) + (1e-5 * p if i < 4 else 0.0)))
        moments.append(m)
    return {"out": out, "loss": loss.reshape(1), "w": new[:4], "b": new[4:], "m": moments}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("session", "stream"):
        rows, cols = (case["n"], case["n"]) if kind == "stream" else (case["rows"], case["cols"])
        counts, ab = _counts(rows, cols, case, case["dose"], seed, case.get("bits", 16))
        ref = _Exact(counts, case, case.get("rotation", 0.0))
        four = tuple(float(np.float32(ab[k])) for k in ("C10", "C12", "phi12")) + (0.0,)
        obj = ref.object(four)
        if kind == "stream":
            return {"phase": obj.angle()}
        return {"object": obj, "loss": float(ref.losses([four])[0][0])} if case["loss"] else {"object": obj}
    if kind in ("score", "terms"):
        counts, _ = _counts(case["rows"], case["cols"], case, 1000.0, seed)
        c = _candidates(case, seed) if kind == "score" else np.concatenate(_terms(case, seed), axis=1)
        loss, means = _Exact(counts, case).losses([tuple(float(v) for v in row) for row in c])
        if kind == "score" and case["n_cand"] == 1 and not case["c30"]:
            return {"phase": means[0], "loss": float(loss[0])}
        return {"loss": loss}
    if kind == "train":
        return _train_exact(case, seed)
    if kind in ("decode", "encode"):
        return None
    stack, shifts = _waves(case, seed)
    s = shifts.double().cuda()
    ramp_r = torch.fft.fftfreq(case["rows"], dtype=torch.float64, device="cuda")[None, :, None] * s[:, 0, None, None]
    ramp_c = torch.fft.fftfreq(case["cols"], dtype=torch.float64, device="cuda")[None, None, :] * s[:, 1, None, None]
    moved = torch.fft.ifft2(torch.fft.fft2(stack.to(torch.complex128))
                            * torch.polar(torch.ones_like(ramp_r), -2 * math.pi * ramp_r)
                            * torch.polar(torch.ones_like(ramp_c), -2 * math.pi * ramp_c))
    if case["reference"]:
        over = (moved * moved[:1].conj()).sum(dim=(1, 2), keepdim=True)
        moved = moved * (over.conj() / over.abs())
    joined = moved.mean(dim=0)
    return {"joined": joined, "aligned": moved} if case["aligned"] else {"joined": joined}
