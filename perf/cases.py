"""What a user of this framework has it do, as measurable cases.

listed()            the cases, draw(rng) one more of the same ranges
prepare(case, seed) the movie, the plan and the output buffers a program holds
run(state)          one pass through the public entry points
work(case)          bytes and operations one pass cannot do without
exact(case, seed)   the same outputs in 64 bits from plain torch

Kinds of pass:
  run        a whole movie whose frames are on the GPU (Plan.run)
  host       a whole movie whose frames are in pinned host memory (Plan.run_host)
  windows    forward transforms and pair stage, up to the correlation windows
             of every frame pair (Plan.forward, Plan.pairs)
  objective  value and gradient of the frame-to-sum objective at given shifts,
             forward and backward through autograd (autograd.sum_objective)
  batch      several movies of uneven size and depth in one call (Batch.run)

Whole movies (run, host, batch) drift by whole pixels of the aligned image and
hold many counts, so that each pair's peak lies in the middle of a cell of the
1/32-px grid of the peak search: with a peak on the edge between two cells the
last bit of a window would decide between two shifts 1/32 px apart, and an
image of one could not be compared with an image of the other.  The other
kinds have sub-pixel drift and counting doses.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from motioncorr1exp_b200 import _lib, api
from motioncorr1exp_b200.autograd import sum_objective

# pixel types: MRC mode, torch type of the stored pixels, largest count
PIXELS = {
    "i8": (0, torch.uint8, 127),
    "u8": (api.MODE_U8, torch.uint8, 255),
    "i16": (1, torch.int16, 32767),
    "u16": (6, torch.uint16, 65535),
    "f32": (2, torch.float32, 1 << 24),
    "f16": (api.MODE_F16, torch.float16, 2048),
}
BFACTOR = 150.0


def _case(name, kind, nx, ny, frames, pixel, mean, **options):
    """Every field of a case; `side` is the square crop (0: the smaller side)."""
    c = dict(name=name, kind=kind, nx=nx, ny=ny, frames=frames, pixel=pixel, mean=mean, side=0, bin=1, fod=2, pbx=96,
             refs=False, itr=0, refine=False, movies=1)
    c.update(options)
    return c


def listed():
    return [
        # a quick check on a small crop: latency and launches
        _case("run_256", "run", 264, 256, 8, "u16", 1000.0, pbx=64),
        # the benchmark's small movie: 16 float frames of 1024^2
        _case("run_1024", "run", 1024, 1024, 16, "f32", 400.0),
        # the benchmark's counting movie, stage by stage up to the windows
        _case("windows_3710", "windows", 3838, 3710, 40, "i8", 1.2, fod=7),
        # the same movie as a program gets it: frames in pinned host memory,
        # image back on the host
        _case("host_3710", "host", 3838, 3710, 40, "u8", 60.0, fod=7),
        # the same detector with dark and gain references, a short movie
        _case("windows_refs", "windows", 3838, 3710, 16, "u16", 20.0, fod=2, refs=True),
        # the benchmark's super-resolution movie (fewer frames), binned by two
        _case("run_bin2", "run", 7676, 7420, 24, "u8", 30.0, bin=2),
        # the benchmark's float movie with one realignment round and the
        # gradient refinement
        _case("run_refine", "run", 4096, 4096, 24, "f32", 100.0, itr=1, refine=True),
        # one evaluation of the refinement's objective and gradient, 60 frames
        _case("objective_4096", "objective", 4096, 4096, 60, "f32", 1.0),
        # a wide detector whose square crop has awkward factors (4 x 3 x 11 x 31)
        _case("windows_4092", "windows", 5760, 4092, 16, "u8", 1.5),
        # an odd-sized user crop of a square detector, half-precision frames
        _case("run_crop1500", "run", 2048, 2048, 24, "f16", 200.0, side=1500),
        # small ragged frames, few counts, narrow search box
        _case("windows_520", "windows", 530, 520, 30, "i16", 2.0, pbx=64),
        # a facility's queue: six movies of uneven size and depth
        _case("batch_mixed", "batch", 2048, 2048, 20, "u8", 60.0, fod=4, movies=6),
    ]


def _max_prime(n):
    p, best = 2, 1
    while p * p <= n:
        while n % p == 0:
            best, n = p, n // p
        p += 1
    return max(best, n)


def draw(rng):
    """One more case: any kind, sides spread over their logarithm from 240 to
    4096 (even, ragged frames around them, no prime factor above 127), depths
    from 6 to 48, every pixel type; the pixels of a movie are bounded so that
    no drawn case costs more than the largest listed one."""
    kind = rng.choice(["run", "run", "windows", "windows", "host", "objective", "batch"])
    while True:
        n = 2 * int(round(math.exp(rng.uniform(math.log(120), math.log(2048)))))
        if _max_prime(n) <= 127:
            break
    if kind == "batch":
        n = min(n, 1600)
        while _max_prime(n) > 127:
            n += 2
    bin_ = 2 if kind in ("run", "windows") and n <= 2400 and rng.random() < 0.2 else 1
    side = n * bin_
    frames = int(round(math.exp(rng.uniform(math.log(6), math.log(48)))))
    frames = max(6, min(frames, int(2.4e8 / (side * side)), int(6e9 / (n * n * frames))))
    crop = rng.random() < 0.3
    nx = side + rng.randrange(0, 2 * (side // 16) + 1)
    ny = side + (rng.randrange(1, side // 16 + 1) if crop else 0)
    pixel = rng.choice(list(PIXELS))
    if kind in ("run", "host", "batch"):
        pixel = rng.choice(["u16", "f32", "i16"] if n < 1400 else ["u8", "u16", "f32", "f16"])
        mean = {"u8": 60.0, "f16": 200.0}.get(pixel, 1000.0 if n < 1400 else 300.0)
    else:
        mean = round(math.exp(rng.uniform(math.log(0.8), math.log(20.0))), 2)
    return _case("drawn", kind, nx, ny, frames, pixel, mean, side=side if crop else 0, bin=bin_,
                 fod=rng.choice([0, 1, 2]) if frames < 16 else rng.choice([2, 4, 7]),
                 pbx=rng.choice([64, 96, 96, 128]),
                 refs=kind == "windows" and rng.random() < 0.25,
                 itr=rng.choice([0, 0, 0, 1, 2]) if kind == "run" else 0,
                 movies=rng.randrange(3, 7) if kind == "batch" else 1)


# ------------------------------------------------------------------ geometry --
def _movies(case):
    """The movies of a case: itself, or the uneven queue of a batch."""
    if case["kind"] != "batch":
        return [case]
    out = []
    for m in range(case["movies"]):
        # every other movie half the size, depths from the full one down
        nx, ny = (case["nx"], case["ny"]) if m % 2 == 0 else (case["nx"] // 2, case["ny"] // 2)
        side = case["side"] if m % 2 == 0 else case["side"] // 4 * 2
        out.append(dict(case, nx=nx, ny=ny, side=side, frames=max(6, case["frames"] - 2 * m)))
    return out


def _sides(case):
    """(crop side, aligned side) as the framework takes them."""
    nu = case["side"] or min(case["nx"], case["ny"])
    nu = min(nu, case["nx"], case["ny"])
    nu = nu // 4 * 4 if case["bin"] == 2 else nu // 2 * 2
    return nu, nu // case["bin"] // 2 * 2


def _params(case):
    nf = case["frames"]
    p = api.Params(crop_nsam=case["side"], bin=float(case["bin"]), nEnd=nf - 1, nEndSum=nf - 1, bfactor=BFACTOR,
                   CCPeakSearchDim=case["pbx"], FrameDistOffset=min(case["fod"], nf // 2 - 1), iter=case["itr"],
                   refine=int(case["refine"]))
    return api.verify_params(p, nf)


def _pairs(case):
    nf = case["frames"]
    dist = max(1, nf // 2 - min(case["fod"], nf // 2 - 1))
    return [(i, j) for i in range(nf) for j in range(i + dist, nf)]


# -------------------------------------------------------------------- inputs --
def _movie(case, seed):
    """Frames (frames, ny, nx) on the GPU and the drift of each in raw pixels:
    a low-passed random field plus Gaussian blobs, drifting along a random walk
    with a linear trend, Poisson counts."""
    nf, ny, nx = case["frames"], case["ny"], case["nx"]
    whole = case["kind"] in ("run", "host", "batch")
    rng = np.random.Generator(np.random.PCG64(seed))
    ang = rng.uniform(0, 2 * math.pi)
    steps = rng.normal(0.0, 0.5, (nf, 2)) + 0.4 * np.array([math.cos(ang), math.sin(ang)])
    track = np.cumsum(steps, 0) * case["bin"]
    track -= track[0]
    grid = float(case["bin"]) if whole else 0.25
    track = np.rint(track / grid) * grid
    whole_px = np.floor(track)
    pad = 16 + int(np.abs(track).max())
    cy, cx = (-(-(v + 2 * pad) // 128) * 128 for v in (ny, nx))
    g = torch.Generator(device="cuda").manual_seed(seed)
    fy = torch.fft.fftfreq(cy, device="cuda")[:, None]
    fx = torch.fft.rfftfreq(cx, device="cuda")[None, :]
    f2 = fy * fy + fx * fx
    F = torch.fft.rfft2(torch.randn((cy, cx), generator=g, device="cuda")) * (f2 <= (0.1 / case["bin"]) ** 2)
    F *= math.sqrt(cy * cx) / torch.linalg.vector_norm(torch.fft.irfft2(F, s=(cy, cx)))
    dots = torch.zeros(cy * cx, device="cuda")
    at = torch.randint(0, cy * cx, (max(8, cy * cx // 5000),), generator=g, device="cuda")
    dots.index_fill_(0, at, 2.0 * 2 * math.pi * 36.0)
    F += torch.fft.rfft2(dots.view(cy, cx)) * torch.exp(-2.0 * math.pi ** 2 * 36.0 * f2)
    mode, dtype, most = PIXELS[case["pixel"]]
    out = torch.empty((nf, ny, nx), dtype=dtype, device="cuda")
    shifted = {}
    for k in range(nf):
        frac = tuple(track[k] - whole_px[k])
        if frac not in shifted:
            ph = torch.exp(-2j * math.pi * (fx * frac[0] + fy * frac[1])) if any(frac) else 1.0
            shifted[frac] = case["mean"] * torch.clamp(1.0 + 0.4 * torch.fft.irfft2(F * ph, s=(cy, cx)), min=0.0)
        dx, dy = (int(v) for v in whole_px[k])
        rate = shifted[frac][pad - dy:pad - dy + ny, pad - dx:pad - dx + nx]
        out[k] = torch.poisson(rate.contiguous(), generator=g).clamp_(max=most).to(dtype)
    return out, track


def _references(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 7))
    shape = (case["ny"], case["nx"])
    dark = rng.random(shape, dtype=np.float32) * 0.5
    gain = 0.9 + 0.2 * rng.random(shape, dtype=np.float32)
    return dark, gain


def _trial_shifts(case, track, seed):
    """Sum shifts a refinement would try: the drift, off by ~0.2 px."""
    rng = np.random.Generator(np.random.PCG64(seed + 11))
    return torch.tensor(track + rng.normal(0.0, 0.2, track.shape), dtype=torch.float32)


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    if case["kind"] == "batch":
        movies, keep = [], []
        for m, c in enumerate(_movies(case)):
            frames, _ = _movie(c, seed + 1000 * m)
            n = _sides(c)[1]
            keep.append(frames)
            movies.append(dict(params=_params(c), nx=c["nx"], ny=c["ny"], nz=c["frames"], mode=PIXELS[c["pixel"]][0],
                               device_ptr=frames.data_ptr(), image=_pinned(n, n).numpy(),
                               frame_shifts=np.empty((c["frames"], 2))))
        torch.cuda.synchronize()
        return dict(kind="batch", batch=api.Batch(lanes=2), movies=movies, keep=keep)
    frames, track = _movie(case, seed)
    mode = PIXELS[case["pixel"]][0]
    plan = api.Plan(_params(case), case["nx"], case["ny"], case["frames"], mode)
    state = dict(kind=case["kind"], plan=plan, refine=case["refine"])
    if case["refs"]:
        dark, gain = _references(case, seed)
        plan.set_refs(dark=dark, norm=gain)
    torch.cuda.synchronize()
    if case["kind"] == "host":
        state["frames"] = torch.empty(frames.shape, dtype=frames.dtype, pin_memory=True).copy_(frames).numpy()
    else:
        state["keep"] = frames
        plan.bind_frames_device(frames.data_ptr())
    if case["kind"] in ("run", "host"):
        state["image"] = _pinned(plan.nsam, plan.nsam).numpy()
    elif case["kind"] == "windows":
        state["windows"] = _pinned(plan.npairs, case["pbx"], case["pbx"])
    else:
        plan.forward()
        state["shifts"] = _trial_shifts(case, track, seed)
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run(state["movies"])
        return [{"image": m["image"], "frame_shifts": m["frame_shifts"]} for m in state["movies"]]
    plan = state["plan"]
    if kind == "objective":
        shifts = state["shifts"].detach().requires_grad_(True)
        value = sum_objective(shifts, plan)
        value.backward()
        return {"value": value.detach(), "gradient": shifts.grad}
    if kind == "windows":
        plan.forward()
        plan.pairs()
        # the C ABI's getter, into the program's pinned buffer
        _lib.check(_lib.lib().mc_plan_get_boxes(plan.handle, state["windows"].data_ptr()))
        return {"windows": state["windows"], "cc": plan.pair_results()["cc"], "means": plan.frame_means()}
    if kind == "host":
        image = plan.run_host(state["frames"], out=state["image"])
    else:
        image = plan.run(out=state["image"])
    shifts = plan.frame_shifts()
    # refined shifts are the end of an iteration, known to its last step
    return {"image": image, "frame_shifts": shifts.astype(np.float32) if state["refine"] else shifts}


# ---------------------------------------------------------------------- work --
def work(case):
    """Raw pixels read once and outputs written once; operations of the real
    transforms (5/2 N log2 N), of each pair's cross power and inverse transform
    onto the search box, and of the phase-shifted sum."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _movies(case):
        nu, n = _sides(c)
        nf, half = c["frames"], (n // 2 + 1) * n
        forward = nf * (2.5 * nu * nu * math.log2(float(nu) * nu))
        pairs = len(_pairs(c)) + c["frames"] * c["itr"]
        pair = half * (8.0 + 5.0 * math.log2(c["pbx"]))
        shift_sum = nf * half * 8.0
        image = 4.0 * n * n
        raw = float(nf) * nu * nu * torch.empty((), dtype=PIXELS[c["pixel"]][1]).element_size()
        if c["kind"] == "objective":
            total["bytes"] += nf * half * 8.0
            total["flops"] += shift_sum + nf * half * 20.0
        elif c["kind"] == "windows":
            total["bytes"] += raw + (8.0 * nu * nu if c["refs"] else 0.0) + 4.0 * pairs * c["pbx"] ** 2
            total["flops"] += forward * (2 if c["refs"] else 1) + pairs * pair
        else:
            total["bytes"] += raw + image
            total["flops"] += (forward + pairs * pair + shift_sum * (1 + c["itr"] + (1 if c["refine"] else 0)) +
                               2.5 * n * n * math.log2(float(n) * n))
            if c["refine"]:
                total["flops"] += nf * half * 20.0
    return total


# -------------------------------------------------------- the same in 64 bits --
def _signed(n):
    """Signed index along ky: k below n/2, k - n from there on."""
    k = torch.arange(n, device="cuda")
    return torch.where(k < n // 2, k, k - n).double()


def _spectra64(case, frames, refs=None, second=False):
    """Half spectra [frame][ky][kx] of the crops, Fourier-cropped when binned."""
    nu, n = _sides(case)
    out = torch.empty((case["frames"], n, n // 2 + 1), dtype=torch.complex128, device="cuda")
    for k in range(case["frames"]):
        x = frames[k, :nu, :nu].to(torch.float64)
        if refs is not None and not second:
            dark, gain = (torch.from_numpy(r[:nu, :nu]).cuda().double() for r in refs)
            x = (x - dark) * gain
        F = torch.fft.rfft2(x)
        out[k, :n // 2] = F[:n // 2, :n // 2 + 1]
        out[k, n // 2:] = F[nu - n // 2:, :n // 2 + 1]
    return out


def _weight64(n):
    kx = torch.arange(n // 2 + 1, device="cuda").double()
    return torch.exp(-0.5 * BFACTOR / n / n * (_signed(n)[:, None] ** 2 + kx[None, :] ** 2))


def _windows64(A, B, pairs, n, pbx):
    """Correlation windows around zero lag, rows y and columns x from -pbx/2."""
    lag = torch.arange(pbx, device="cuda").double() - pbx // 2
    kx = torch.arange(n // 2 + 1, device="cuda").double()
    h = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    h[0] = h[-1] = 1.0
    ey = torch.exp(2j * math.pi / n * torch.remainder(lag[:, None] * _signed(n)[None, :], n))
    ex = h[:, None] * torch.exp(2j * math.pi / n * torch.remainder(kx[:, None] * lag[None, :], n))
    w = _weight64(n) / ((n // 2 + 1.0) * n)
    out = torch.empty((len(pairs), pbx, pbx), dtype=torch.float64, device="cuda")
    for p, (i, j) in enumerate(pairs):
        out[p] = ((ey @ (A[i] * B[j].conj() * w)) @ ex).real
    return out


def _peaks64(windows, n):
    """Shift and correlation of each window: the integer peak, the 16 x 16 box
    around it, cosine-masked and Fourier-upsampled by 32, the largest value."""
    P, pbx, _ = windows.shape
    hb = pbx // 2
    at = windows.reshape(P, -1).argmax(1).cpu().numpy()
    oy, ox = (np.clip(v - 8, 0, pbx - 16) for v in (at // pbx, at % pbx))
    ky, kx = np.meshgrid(np.r_[0:8, -8:0], np.arange(9), indexing="ij")
    r = np.floor(np.sqrt(ky * ky + kx * kx))
    mask = torch.from_numpy(np.where(r < 8, np.cos(r * math.pi / 8) / 2 + 0.5, 0.0)).cuda()
    shift, cc = np.empty((P, 2)), np.empty(P)
    for p in range(P):
        S = torch.fft.rfft2(windows[p, oy[p]:oy[p] + 16, ox[p]:ox[p] + 16]) * mask
        pad = torch.zeros((512, 257), dtype=torch.complex128, device="cuda")
        pad[:8, :9], pad[504:, :9] = S[:8], S[8:]
        up = torch.fft.irfft2(pad, s=(512, 512), norm="forward")
        m = int(up.argmax())
        shift[p] = ox[p] + (m % 512) / 32 - hb, oy[p] + (m // 512) / 32 - hb
        cc[p] = float(up.view(-1)[m]) / n / n / 256
    return shift, cc


def _solve64(case, pairs, shift):
    """Per-step shifts by least squares; None where the threshold on the
    residuals would drop a pair."""
    M = np.zeros((len(pairs), case["frames"] - 1))
    for r, (i, j) in enumerate(pairs):
        M[r, i:j] = 1.0
    s = np.linalg.lstsq(M, shift, rcond=None)[0]
    return s if np.abs(M @ s - shift).max() < 0.7 else None


def _sum64(F, shifts, n):
    """Sum of the spectra, each shifted by (x, y) pixels."""
    kx = torch.arange(n // 2 + 1, device="cuda").double()
    S = torch.zeros_like(F[0])
    for k, (sx, sy) in enumerate(shifts):
        S += F[k] * torch.exp(2j * math.pi / n * float(sy) * _signed(n))[:, None] * torch.exp(2j * math.pi / n * float(sx) * kx)
    return S


def _objective64(F, shifts, n):
    """Objective, gradient and 2x2 Hessian blocks of the frame-to-sum correlation."""
    kx = torch.arange(n // 2 + 1, device="cuda").double()
    h = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    h[0] = h[-1] = 1.0
    hw = _weight64(n) * h
    S = _sum64(F, shifts, n)
    wx, wy = 2 * math.pi / n * kx[None, :], 2 * math.pi / n * _signed(n)[:, None]
    grad, hess = np.empty((len(shifts), 2)), np.empty((len(shifts), 3))
    for k in range(len(shifts)):
        P = _sum64(F[k:k + 1], shifts[k:k + 1], n)
        u = hw * ((S - P).conj() * P)
        grad[k] = [-2 * float((u.imag * w).sum()) for w in (wx, wy)]
        hess[k] = [-2 * float((u.real * w).sum()) for w in (wx * wx, wx * wy, wy * wy)]
    return float((hw * (S.real ** 2 + S.imag ** 2)).sum()), grad, hess


def _refine64(F, s, n):
    """The refinement's block-Newton steps from the sum shifts `s`."""
    for _ in range(4):
        _, g, H = _objective64(F, s, n)
        det = H[:, 0] * H[:, 2] - H[:, 1] ** 2
        d = -np.stack([H[:, 2] * g[:, 0] - H[:, 1] * g[:, 1], H[:, 0] * g[:, 1] - H[:, 1] * g[:, 0]], 1) / det[:, None]
        s = s + d
        if np.hypot(*d.T).max() < 1e-4:
            break
    return s


def _whole64(case, seed):
    n, nf = _sides(case)[1], case["frames"]
    frames, _ = _movie(case, seed)
    F = _spectra64(case, frames)
    pairs = _pairs(case)
    step = _solve64(case, pairs, _peaks64(_windows64(F, F, pairs, n, case["pbx"]), n)[0])
    if step is None:
        return None
    total = np.concatenate([np.zeros((1, 2)), np.cumsum(step, 0)])
    for _ in range(case["itr"]):
        S = _sum64(F, -total, n)
        total = _peaks64(_windows64(S[None], F, [(0, k) for k in range(nf)], n, case["pbx"]), n)[0]
        total = total - total[0]
    if case["refine"]:
        s = _refine64(F, -total, n)
        total = s[0] - s
    middle = total[min(nf // 2 + 1, nf - 1)]
    image = torch.fft.irfft2(_sum64(F, middle - total, n), s=(n, n))
    return {"image": image, "frame_shifts": total}


def exact(case, seed):
    n = _sides(case)[1]
    if case["kind"] == "batch":
        return [_whole64(c, seed + 1000 * m) for m, c in enumerate(_movies(case))]
    if case["kind"] in ("run", "host"):
        return _whole64(case, seed)
    frames, track = _movie(case, seed)
    if case["kind"] == "objective":
        shifts = _trial_shifts(case, track, seed).double().numpy()
        value, grad, _ = _objective64(_spectra64(case, frames), shifts, n)
        return {"value": value, "gradient": torch.from_numpy(grad)}
    refs = _references(case, seed) if case["refs"] else None
    A = _spectra64(case, frames, refs)
    B = _spectra64(case, frames, refs, second=True) if case["refs"] else A
    windows = _windows64(A, B, _pairs(case), n, case["pbx"])
    # each window's correlation is the largest value of its upsampled peak
    return {"windows": windows, "cc": _peaks64(windows, n)[1], "means": A[:, 0, 0].real / n / n}
