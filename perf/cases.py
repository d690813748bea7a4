"""The work that users of this library have it do, as cases that can be timed: exit waves and HRTEM images, STEM and
4D-STEM scans on the grids in use (powers of two, 3 and 5 times a power of two, 500 = 4 * 5^3, odd lengths), frozen
phonons, job tables, the waves detector, the learned potential profile's two directions and scan post-processing.

A case names its kind, grid and counts; `prepare` makes what a program holds before the call, `run` is one pass through
the public entry points, `exact` the same result in float64 with torch alone. Waves and measurements are float32
results that the boundary widens to float64; they are returned as the float32 / complex64 arrays a program stores."""

import json
import math
import os

import numpy as np
import torch

import simulatokit_b200 as sk
from simulatokit_b200 import _lib as L

SRTIO3 = (3.905, [(38, 0, 0, 0), (22, .5, .5, .5), (8, .5, .5, 0), (8, .5, 0, .5), (8, 0, .5, .5)])
SILICON = (5.431, [(14, *f) for f in ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0), (.25, .25, .25),
                                      (.25, .75, .75), (.75, .25, .75), (.75, .75, .25))])
SAMPLING = 0.061  # [A / pixel], the headline scan's (31.24 A on 512 points)
TABLE = [256, 384, 500, 640]  # job tables: grid sides
ELEMENTS = [6, 8, 14, 79]  # the amorphous cell's


def listed():
    return [
        # the smallest call: one plane wave through a thin, already sliced crystal (latency, launches, host work)
        {"name": "run_128", "kind": "run", "nx": 128, "ny": 128, "slices": 4},
        # one HRTEM image from a structure: potential, exit wave, objective lens (10 slices of half a cell)
        {"name": "hrtem_256", "kind": "hrtem", "nx": 256, "ny": 256, "slices": 10},
        # a small scan with the common detectors on a thin crystal
        {"name": "scan_256", "kind": "scan", "nx": 256, "ny": 256, "slices": 10, "px": 16, "py": 16,
         "detectors": "annular com", "form": "fused"},
        # the headline: 64 x 64 BF + HAADF scan, 20 slices
        {"name": "scan_512", "kind": "scan", "nx": 512, "ny": 512, "slices": 20, "px": 64, "py": 64,
         "detectors": "annular", "form": "fused"},
        # a large field of view: 1024^2, fewer positions
        {"name": "scan_1024", "kind": "scan", "nx": 1024, "ny": 1024, "slices": 20, "px": 16, "py": 16,
         "detectors": "annular", "form": "fused"},
        # a grid chosen by its sampling, not for its transform: 500 = 4 * 5^3, segmented detector beside the annular ones
        {"name": "scan_500", "kind": "scan", "nx": 500, "ny": 500, "slices": 10, "px": 12, "py": 12,
         "detectors": "annular segmented", "form": "fused"},
        # 4D-STEM averaged over frozen phonons: a new potential per configuration, binned patterns and
        # annular images
        {"name": "phonons_768", "kind": "phonons", "nx": 768, "ny": 768, "slices": 16, "px": 8, "py": 8,
         "configurations": 2},
        # the tensor-core form of a scan
        {"name": "bf16x3_512", "kind": "scan", "nx": 512, "ny": 512, "slices": 10, "px": 16, "py": 16,
         "detectors": "annular", "form": "bf16x3"},
        # independent multislice jobs on four grid shapes in one call, each potential its own
        {"name": "jobs_24", "kind": "jobs", "jobs": 24, "most_slices": 40},
        # exit waves of a small scan on an odd grid (331 is prime), resampled to what a program keeps
        {"name": "waves_331x250", "kind": "waves", "nx": 331, "ny": 250, "slices": 6, "px": 4, "py": 4, "rows": 128,
         "columns": 128},
        # the learned finite-projection profile: a training batch's gradients, and inference over profile tables
        {"name": "surrogate", "kind": "surrogate", "batch": 4096, "queries": 100000},
        # a finished 4D-STEM measurement: finite source size, then counting noise, on the device
        {"name": "post_32", "kind": "post", "px": 32, "py": 32, "values": 4096, "sigma": 0.4, "dose": 4000.0},
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def side(b=1024):
        usual = [n for n in (128, 160, 192, 200, 240, 250, 256, 300, 320, 360, 384, 400, 450, 480, 500, 512, 576, 600,
                             640, 720, 750, 768, 800, 900, 960, 1000, 1024) if n <= b]
        pick = rng.random()
        return rng.choice(usual) if pick < 0.6 else 2 * log_int(60, b // 2) if pick < 0.85 else 2 * log_int(50, b // 2) - 1

    def positions(nx, ny, slices, most):
        n = max(1, min(int(most / (nx * ny * slices)), 1024))
        px = log_int(1, min(32, n))
        return px, max(1, min(32, rng.randint(1, max(1, n // px))))

    kind = rng.choice(["scan", "scan", "scan", "scan", "run", "hrtem", "phonons", "jobs", "waves", "surrogate", "post"])
    if kind == "run":
        return {"kind": kind, "nx": side(), "ny": side(), "slices": log_int(2, 32)}
    if kind == "hrtem":
        return {"kind": kind, "nx": side(), "ny": side(), "slices": log_int(4, 32)}
    if kind == "scan":
        form = rng.choice(["fused", "fused", "fused", "bf16x3"])
        nx, ny = (rng.choice([256, 512, 768, 1024]) for _ in range(2)) if form == "bf16x3" else (side(), side())
        if rng.random() < 0.5:
            ny = nx
        slices = log_int(4, 32)
        px, py = positions(nx, ny, slices, 1.5e9)
        return {"kind": kind, "nx": nx, "ny": ny, "slices": slices, "px": px, "py": py, "form": form,
                "detectors": rng.choice(["annular", "annular", "annular segmented", "pixelated", "annular binned"])}
    if kind == "phonons":
        n, slices = rng.choice([256, 384, 500, 512, 640, 768]), 4 * log_int(1, 6)
        px, py = positions(n, n, slices, 3e8)
        return {"kind": kind, "nx": n, "ny": n, "slices": slices, "px": min(px, 12), "py": min(py, 12),
                "configurations": rng.randint(1, 3)}
    if kind == "jobs":
        return {"kind": kind, "jobs": rng.randint(4, 24), "most_slices": rng.randint(12, 40)}
    if kind == "waves":
        nx, ny, slices = side(512), side(512), log_int(3, 12)
        px, py = positions(nx, ny, slices, 2e7)
        return {"kind": kind, "nx": nx, "ny": ny, "slices": slices, "px": min(px, 6), "py": min(py, 6),
                "rows": rng.randint(32, 300), "columns": rng.randint(32, 300)}
    if kind == "surrogate":
        return {"kind": kind, "batch": log_int(512, 8192), "queries": log_int(4000, 200000)}
    return {"kind": kind, "px": log_int(8, 40), "py": log_int(8, 40), "values": log_int(16, 4096),
            "sigma": round(rng.uniform(0.1, 0.6), 2), "dose": float(log_int(300, 30000))}


# ---- what a program has in hand before the call ----------------------------------------------------------------------

def crystal(kind, nx, ny, slices, per_slice, rng):
    """A thermally displaced crystal (rms 0.06 A an axis) of whole cells near the sampling: (box, numbers, positions,
    slice thickness), `per_slice` cells along the beam to a slice."""
    a, cell = kind
    m = [max(1, round(n * SAMPLING / a)) for n in (nx, ny)] + [math.ceil(slices * per_slice)]
    frac = np.array([c[1:] for c in cell])
    shifts = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), axis=-1).reshape(-1, 3)
    ideal = ((shifts[:, None, :] + frac) * a).reshape(-1, 3)
    box = np.array(m) * a
    box[2] = slices * per_slice * a
    keep = ideal[:, 2] < box[2] - 1e-6
    ideal, numbers = ideal[keep], np.tile([c[0] for c in cell], len(shifts))[keep]
    return box, numbers, ideal, rng.normal(0.0, 0.06, ideal.shape), per_slice * a


def model(case, seed):
    """Everything random about a case, as numbers: what both `prepare` and `exact` start from."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    m = {"defocus": float(rng.uniform(-60, 60)), "shift": rng.uniform(0, 1, 2)}
    if kind in ("run", "scan", "waves", "hrtem"):
        box, z, ideal, d, dz = crystal(SRTIO3, case["nx"], case["ny"], case["slices"], 0.5 if kind == "hrtem" else 1.0, rng)
        m.update(box=box, numbers=z, positions=np.mod(ideal + d, box), dz=dz)
    elif kind == "phonons":
        box, z, ideal, _, dz = crystal(SILICON, case["nx"], case["ny"], case["slices"], 0.25, rng)
        m.update(box=box, numbers=z, positions=ideal, dz=dz,
                 displacements=[rng.normal(0.0, 0.075, ideal.shape) for _ in range(case["configurations"])])
    elif kind == "jobs":
        m["jobs"], shapes = [], np.random.default_rng(case["jobs"])  # the table's shapes are the case's own
        for j in range(case["jobs"]):
            n = TABLE[int(shapes.integers(4))]
            slices = int(shapes.integers(min(10, case["most_slices"]), case["most_slices"] + 1))
            side = rng.uniform(20, 40, 2)
            dz = rng.uniform(1, 2)
            atoms = int(0.02 * side[0] * side[1] * slices * dz)
            box = np.array([side[0], side[1], slices * dz])
            m["jobs"].append({"n": n, "slices": slices, "box": box, "dz": dz, "numbers": rng.integers(1, 81, atoms),
                              "positions": rng.uniform(0, 1, (atoms, 3)) * box, "energy": float(rng.uniform(80e3, 300e3)),
                              "at": tuple(rng.uniform(0, 1, 2) * side) if j % 2 else None})
    elif kind == "surrogate":
        m["parameters"] = np.concatenate([rng.normal(0, s, k) for k, s in (
            (103 * 16, .5), (64 * 18, .3), (64, .1), (4096, .15), (64, .1), (4096, .15), (64, .1), (64, .15), (1, .1))]
        ).astype(np.float32)
        for name, n in (("batch", case["batch"]), ("queries", case["queries"])):
            zl = rng.uniform(-4, 3, n)
            m[name] = (rng.choice(ELEMENTS, n).astype(np.int32), np.exp(rng.uniform(math.log(0.05), math.log(5.0), n)),
                       zl, zl + rng.uniform(0.2, 1.5, n))
        m["target"] = rng.uniform(0, 1, case["batch"])
    return m


def potential(m, case):
    return sk.Potential(sk.AtomicStructure(m["box"], m["numbers"], m["positions"]), case["nx"], case["ny"],
                        slice_thicknesses=[m["dz"]] * case["slices"])


def probe_and_scan(m, case):
    energy, semiangle = (300e3, 25.0) if case["kind"] == "phonons" else (200e3, 20.0)
    grid = sk.Grid(case["nx"], case["ny"], float(m["box"][0]), float(m["box"][1]))
    probe = sk.Probe(sk.ElectronBeam(energy), grid, sk.Aperture(semiangle), sk.Aberrations(C10=m["defocus"], C30=1e4))
    cell = SILICON[0] if case["kind"] == "phonons" else SRTIO3[0]
    start = m["shift"] * cell
    return probe, sk.GridScan(tuple(start), tuple(start + cell), case["px"], case["py"])


def binned_window(case, m, lam):
    """Half-width [mrad] of the binned patterns: 60, or what the grid reaches."""
    reach = min(case["nx"] // 2 / m["box"][0], case["ny"] // 2 / m["box"][1]) * lam * 1e3
    return min(60.0, 0.9 * reach)


def detectors(case, m, probe):
    # (a centre of mass is a small difference of large float32 sums on a centred thin crystal: one listed case has it)
    words = "annular binned" if case["kind"] == "phonons" else case["detectors"]
    made = []
    for w in words.split():
        made += {"annular": lambda: [sk.AnnularDetector(0, 20), sk.AnnularDetector(50, 120)],
                 "com": lambda: [sk.CenterOfMassDetector()],
                 "segmented": lambda: [sk.SegmentedDetector(2, 4, 20, 90, 0.1)],
                 "pixelated": lambda: [sk.PixelatedDetector("valid")],
                 "binned": lambda: [sk.BinnedPixelatedDetector(binned_window(case, m, probe.beam.wavelength), (128, 128))],
                 }[w]()
    return made


def prepare(case, seed):
    m, kind = model(case, seed), case["kind"]
    engine = sk.Engine.require()
    state = {"case": case, "engine": engine}
    if kind in ("run", "hrtem"):
        beam = sk.ElectronBeam(200e3)
        grid = sk.Grid(case["nx"], case["ny"], float(m["box"][0]), float(m["box"][1]))
        state["wave"] = sk.Waves.plane_wave(beam, grid)
    if kind == "run":
        state["potential"] = potential(m, case)
        state["potential"].handle(engine)
    elif kind == "hrtem":
        state["model"] = m
        state["lens"] = sk.ContrastTransferFunction(sk.Aberrations(C10=m["defocus"], C30=1e7), 20.0, True, 30.0, 0.1)
    elif kind in ("scan", "waves"):
        state["potential"] = potential(m, case)
        state["potential"].handle(engine)
        state["probe"], state["scan"] = probe_and_scan(m, case)
        if kind == "scan":
            state["detectors"] = detectors(case, m, state["probe"])
            state["options"] = sk.ExecutionOptions(form=case["form"])
        else:
            state["detectors"] = sk.WavesDetector(case["rows"], case["columns"])
    elif kind == "phonons":
        structure = sk.AtomicStructure(m["box"], m["numbers"], m["positions"])
        state["phonons"] = sk.FrozenPhonons(structure, displacements=m["displacements"])
        state["dz"] = m["dz"] * (1 + 1e-9)
        state["probe"], state["scan"] = probe_and_scan(m, case)
        state["detectors"] = detectors(case, m, state["probe"])
    elif kind == "jobs":
        table = sk.JobTable()
        for j in m["jobs"]:
            p = sk.Potential(sk.AtomicStructure(j["box"], j["numbers"], j["positions"]), j["n"], j["n"],
                             slice_thicknesses=[j["dz"]] * j["slices"])
            p.handle(engine)
            if j["at"] is None:
                table.add_plane_wave(p, j["energy"])
            else:
                table.add_probe(p, sk.Probe(sk.ElectronBeam(j["energy"]), p.grid, sk.Aperture(20.0)), j["at"])
        state["table"] = table
    elif kind == "surrogate":
        net = sk.Surrogate(ELEMENTS, n_samples=4096, steps=1, batch=1024, engine=engine)
        net.parameters(set_to=m["parameters"], mean_std=(0.0, 1.0))
        state.update(net=net, batch=m["batch"], queries=m["queries"], target=m["target"])
    else:
        # what simk_scan_device leaves on the device: float64 patterns, most of the intensity in few pixels
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        n = (case["px"], case["py"], case["values"])
        state["values"] = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) ** 4 * (20.0 / case["values"])
        state["blurred"], state["noisy"] = torch.empty_like(state["values"]), torch.empty_like(state["values"])
        state["seed"] = int(seed)
        torch.cuda.synchronize()
    return state


# ---- one pass --------------------------------------------------------------------------------------------------------

def run(state):
    case, engine = state["case"], state["engine"]
    kind = case["kind"]
    if kind == "run":
        return sk.Multislice.run(state["wave"], state["potential"], engine=engine)[0].field.astype(np.complex64)
    if kind == "hrtem":
        exit_wave = sk.Multislice.run(state["wave"], potential(state["model"], case), engine=engine)[0]
        imaged, image = state["lens"].apply(exit_wave, engine=engine)
        return {"exit": exit_wave.field.astype(np.complex64), "imaged": imaged.field.astype(np.complex64),
                "image": image.astype(np.float32)}
    if kind == "scan":
        got = sk.STEM.scan(state["probe"], [state["potential"]], state["scan"], state["detectors"],
                           options=state["options"], engine=engine)
        return [x.array().astype(np.float32) for x in got]
    if kind == "waves":
        got = sk.STEM.scan(state["probe"], [state["potential"]], state["scan"], state["detectors"], engine=engine)
        return got.array().astype(np.complex64)
    if kind == "phonons":
        got = sk.STEM.scanFrozenPhonons(state["probe"], state["phonons"], case["nx"], case["ny"], state["dz"],
                                        state["scan"], state["detectors"], engine=engine)
        return [x.array().astype(np.float32) for x in got]
    if kind == "jobs":
        return [x.astype(np.float32) for x in state["table"].run(engine=engine)[0]]
    if kind == "surrogate":
        loss, gradients = state["net"].gradients(*state["batch"], state["target"])
        return {"loss": np.float32(loss), "gradients": gradients,
                "profiles": state["net"].evaluate(*state["queries"]).astype(np.float32)}
    v, b, n = state["values"], state["blurred"], state["noisy"]
    at = [L.C.cast(L.C.c_void_p(t.data_ptr()), L.PD) for t in (v, b, n)]
    L.check(engine.lib.simk_gaussian_source_size_device(engine.handle, case["px"], case["py"], case["values"],
                                                        case["sigma"], case["sigma"], 0.2, 0.25, at[0], at[1]))
    L.check(engine.lib.simk_poisson_noise_device(engine.handle, v.numel(), at[1], case["dose"], 1, state["seed"], at[2]))
    return {"blurred": b, "noisy": n}


def work(case):
    """One slice of one wave is two passes over it (a row and a column pass each read and write 8 bytes a point: a wave
    does not fit an SM) and two 2-D transforms; each potential builds V and t by float64 transforms (two of each a
    slice, likewise two passes each)."""
    kind = case["kind"]

    def waves(n, steps):
        return 32.0 * n * steps, steps * (10.0 * n * math.log2(n) + 12.0 * n)

    def built(n, slices):
        return 4 * 64.0 * n * slices, 4 * 5.0 * n * math.log2(n) * slices

    if kind == "post":
        n = case["px"] * case["py"] * case["values"]
        taps = sum(2 * int(4 * case["sigma"] / s + 0.5) + 1 for s in (0.2, 0.25))
        return {"bytes": 48.0 * n, "flops": 2.0 * taps * n}
    if kind == "surrogate":
        net = 2 * (18 * 64 + 2 * 64 * 64 + 64)
        return {"bytes": 36.0 * case["batch"] + 36.0 * case["queries"],
                "flops": 2.0 * net * (3 * case["batch"] + case["queries"])}
    if kind == "jobs":
        n = sum(s * s for s in TABLE) / len(TABLE)
        b, f = waves(n, case["jobs"] * (10 + case["most_slices"]) / 2)
        return {"bytes": b + 12.0 * n * case["jobs"], "flops": f}
    n, slices = case["nx"] * case["ny"], case["slices"]
    b, f = waves(n, slices * case.get("px", 1) * case.get("py", 1) * case.get("configurations", 1))
    if kind in ("hrtem", "phonons"):
        bb, bf = built(n, slices * case.get("configurations", 1))
        b, f = b + bb, f + bf
    if kind == "waves":
        b += 16.0 * case["px"] * case["py"] * case["rows"] * case["columns"]
    return {"bytes": b, "flops": f}


# ---- the same in float64 ---------------------------------------------------------------------------------------------

PLANCK, MASS, LIGHT, CHARGE = 6.62607004e-34, 9.10938356e-31, 299792458.0, 1.6021766208e-19  # CODATA 2014


def wavelength(energy):
    return PLANCK * LIGHT / math.sqrt(energy * (2 * MASS * LIGHT * LIGHT / CHARGE + energy)) / CHARGE * 1e10


def sigma_of(energy):
    kg, coulomb, second = 6.0221408585491615e26, 6.241509125883258e18, 98226947884640.62
    mass = (1 + CHARGE * energy / (MASS * LIGHT ** 2)) * MASS
    return 2 * math.pi * mass * kg * CHARGE * coulomb * wavelength(energy) / (PLANCK * second * coulomb) ** 2


class Field64:
    """Potential, transmission, propagator, probe and detectors of one grid and energy, complex128 on the GPU."""

    def __init__(self, nx, ny, box, energy):
        self.nx, self.ny, self.box, self.lam = nx, ny, box, wavelength(energy)
        self.dx, self.dy, self.energy = box[0] / nx, box[1] / ny, energy
        f = dict(device="cuda", dtype=torch.float64)
        self.kx, self.ky = torch.fft.fftfreq(nx, self.dx, **f)[:, None], torch.fft.fftfreq(ny, self.dy, **f)[None, :]
        self.k2 = self.kx ** 2 + self.ky ** 2
        cut, taper = 0.6666666 / max(self.dx, self.dy) / 2, 0.01 / max(self.dx, self.dy)
        r = torch.sqrt(self.k2)
        ramp = 0.5 * (1 + torch.cos(math.pi * (r - cut + taper) / taper))
        self.limit = torch.where(r > cut, torch.zeros_like(r), torch.where(r > cut - taper, ramp, torch.ones_like(r)))

    def factors(self, numbers):
        """f(k^2) / S(k) of each element."""
        with open(os.path.join(os.path.dirname(L.__file__), "data", "lobato.json")) as f:
            rows = {e["Z"]: e for e in json.load(f)["elements"]}
        a, b = self.kx * self.dx, self.ky * self.dy
        kk = torch.sqrt(a * a + b * b)
        s = torch.where(kk == 0, torch.ones_like(kk), torch.sin(kk) / torch.where(kk == 0, torch.ones_like(kk), kk))
        q, out = 4 * math.pi ** 2 * self.k2, {}
        for z in sorted(set(int(v) for v in numbers)):
            total = torch.zeros_like(q)
            for pa, pb in zip(rows[z]["a"], rows[z]["b"]):
                big_a, big_b = math.pi ** 2 * pa / pb ** 1.5 / 0.0208865737082965, 2 * math.pi / math.sqrt(pb)
                d = q + big_b ** 2
                total += big_a / big_b / d + big_a * big_b / d ** 2
            out[z] = 8 * math.pi * total / (s * self.dx * self.dy)
        return out

    def transmissions(self, numbers, positions, thickness, slices):
        """The bandlimited exp(i sigma V) of every slice."""
        p = np.mod(positions, self.box)
        p[p[:, 2] > self.box[2] - 1e-10, 2] = 0.0
        edges = np.cumsum([thickness] * slices) - 1e-12
        of = np.minimum(np.searchsorted(edges, p[:, 2], side="right"), slices - 1)
        factors, sigma = self.factors(numbers), sigma_of(self.energy)
        fx, fy = p[:, 0] / self.dx, p[:, 1] / self.dy
        ix, iy = np.floor(fx).astype(int), np.floor(fy).astype(int)
        x, y = fx - ix, fy - iy
        for j in range(slices):
            spectrum = 0
            for z, f in factors.items():
                at = np.nonzero((of == j) & (numbers == z))[0]
                if not len(at):
                    continue
                delta = np.zeros((self.nx, self.ny))
                for ox, oy, w in ((0, 0, (1 - x) * (1 - y)), (1, 0, x * (1 - y)), (0, 1, (1 - x) * y), (1, 1, x * y)):
                    np.add.at(delta, ((ix[at] + ox) % self.nx, (iy[at] + oy) % self.ny), w[at])
                spectrum = spectrum + torch.fft.fft2(torch.from_numpy(delta).cuda()) * f
            v = torch.fft.ifft2(spectrum).real if torch.is_tensor(spectrum) else torch.zeros_like(self.k2)
            t = torch.polar(torch.ones_like(v), sigma * v)
            yield torch.fft.ifft2(torch.fft.fft2(t) * self.limit)

    def propagator(self, thickness):
        return torch.polar(self.limit, -math.pi * self.lam * thickness * self.k2)

    def soft_aperture(self, semiangle):
        alpha, phi = torch.sqrt(self.k2) * self.lam, torch.atan2(self.ky.expand_as(self.k2), self.kx.expand_as(self.k2))
        d = torch.sqrt((torch.cos(phi) * self.lam / self.box[0]) ** 2 + (torch.sin(phi) * self.lam / self.box[1]) ** 2)
        a = torch.clamp((semiangle * 1e-3 - alpha) / d + 0.5, 0, 1)
        a[0, 0] = 1.0
        return a

    def chi(self, c10, c30):
        a2 = self.k2 * self.lam ** 2
        return 2 * math.pi / self.lam * (a2 / 2 * c10 + a2 * a2 / 4 * c30)

    def probes(self, semiangle, c10, c30, at):
        spectrum = torch.polar(self.soft_aperture(semiangle), -self.chi(c10, c30))
        spectrum = spectrum / torch.sqrt((spectrum.abs() ** 2).sum())
        x, y = (torch.as_tensor(v, device="cuda", dtype=torch.float64)[:, None] for v in (at[:, 0], at[:, 1]))
        rx, ry = (torch.polar(torch.ones_like(k * v), -2 * math.pi * k * v) for k, v in ((self.kx.T, x), (self.ky, y)))
        return torch.fft.ifft2(spectrum * rx[:, :, None] * ry[:, None, :])

    def exits(self, waves, ts, p):
        """FFT2 of the exit waves of a batch."""
        for j, t in enumerate(ts):
            s = torch.fft.fft2(waves * t) * p
            waves = torch.fft.ifft2(s) if j + 1 < len(ts) else s
        return waves

    def angles(self, nx=None, ny=None):
        return tuple(torch.fft.fftfreq(m, 1.0 / m, device="cuda", dtype=torch.float64) * (self.lam * 1e3 / e)
                     for m, e in ((nx or self.nx, self.box[0]), (ny or self.ny, self.box[1])))

    def cropped(self, region):
        """Kept frequencies along x and y of a 'valid' pattern or a polar region out to `region` mrad."""
        sizes = []
        for n, e, o in ((self.nx, self.box[0], self.lam * 1e3 / self.box[0]), (self.ny, self.box[1], self.lam * 1e3 / self.box[1])):
            if region == "valid":
                m = math.floor(round(2 / 3 / max(self.dx, self.dy) * e, 7))
                m += m % 2 != n % 2
                m = math.floor(round(m / math.sqrt(2), 7))
            else:
                m = int(2 * math.ceil(region / o)) + 1
            sizes.append(min(m + (m % 2 != n % 2), n))
        return [[*range((m + 1) // 2), *range(n - m // 2, n)] for m, n in zip(sizes, (self.nx, self.ny))]

    def detect(self, words, pattern, window):
        """Every detector's values of a batch of patterns, in the order `detectors` makes them."""
        ax, ay = self.angles()
        a2, out = ax[:, None] ** 2 + ay[None, :] ** 2, []
        for w in words.split():
            if w == "annular":
                for i, o in ((0, 20), (50, 120)):
                    out.append((pattern * ((a2 >= i * i) & (a2 < o * o))).sum((1, 2)))
            elif w in ("com", "pixelated"):
                cx, cy = self.cropped("valid")
                p = pattern[:, cx][:, :, cy]
                if w == "pixelated":
                    out.append(torch.fft.fftshift(p, dim=(1, 2)))
                    continue
                kx, ky = (torch.fft.fftfreq(len(c), 1.0 / len(c), device="cuda", dtype=torch.float64) / e
                          for c, e in ((cx, self.box[0]), (cy, self.box[1])))
                out.append(torch.stack([(p * kx[:, None]).sum((1, 2)), (p * ky[None, :]).sum((1, 2))], 1))
            elif w == "segmented":
                cx, cy = self.cropped(90.0)
                p = pattern[:, cx][:, :, cy]
                bx, by = self.angles(len(cx), len(cy))
                alpha = torch.sqrt(bx[:, None] ** 2 + by[None, :] ** 2)
                phi = torch.remainder(torch.atan2(by[None, :].expand_as(alpha), bx[:, None].expand_as(alpha)) - 0.1, 2 * math.pi)
                r = torch.floor(2 * (alpha - 20) / 70)
                az = torch.clamp(torch.floor(4 * (phi / (2 * math.pi))), 0, 3)
                out.append(torch.stack([torch.stack([(p * ((alpha >= 20) & (alpha < 90) & (r == i) & (az == k))).sum((1, 2))
                                                     for k in range(4)], 1) for i in range(2)], 1))
            else:
                edges = torch.linspace(-window, window, 129, device="cuda", dtype=torch.float64)
                wx, wy = (torch.clamp(torch.minimum(edges[1:, None], a + s / 2) - torch.maximum(edges[:-1, None], a - s / 2), min=0) / s
                          for a, s in ((ax, self.lam * 1e3 / self.box[0]), (ay, self.lam * 1e3 / self.box[1])))
                out.append(wx @ pattern @ wy.T)
        return out


def scan_exact(case, m):
    phonons = case["kind"] == "phonons"
    energy, semiangle, dz = (300e3, 25.0, m["box"][2] / case["slices"]) if phonons else (200e3, 20.0, m["dz"])
    field = Field64(case["nx"], case["ny"], m["box"], energy)
    _, scan = probe_and_scan(m, case)
    step = [(scan.end[k] - scan.start[k]) / n for k, n in enumerate((case["px"], case["py"]))]
    at = np.array([(scan.start[0] + i * step[0], scan.start[1] + j * step[1])
                   for i in range(case["px"]) for j in range(case["py"])])
    words = "annular binned" if phonons else case.get("detectors", "")
    total = None
    for d in m.get("displacements", [0.0]):
        ts = list(field.transmissions(m["numbers"], m["positions"] + d, dz, case["slices"]))
        p = field.propagator(dz)
        chunk, got = max(1, int(3e7 / (case["nx"] * case["ny"]))), []
        for first in range(0, len(at), chunk):
            s = field.exits(field.probes(semiangle, m["defocus"], 1e4, at[first:first + chunk]), ts, p)
            if case["kind"] == "waves":
                got.append([resampled(s, case["rows"], case["columns"])])
            else:
                got.append([v.cpu() for v in field.detect(words, s.abs() ** 2, binned_window(case, m, field.lam))])
        values = [torch.cat(v) for v in zip(*got)]
        total = values if total is None else [a + b for a, b in zip(total, values)]
    shape = (case["px"], case["py"])
    if case["kind"] == "waves":
        return total[0].reshape(shape + (case["rows"], case["columns"])).cpu().numpy()
    return [(v / len(m.get("displacements", [0]))).reshape(shape + v.shape[1:]).numpy() for v in total]


def resampled(spectra, rows, columns):
    """The waves of `spectra` on rows x columns points: the lowest frequencies kept, or zeros above them."""
    b, nx, ny = spectra.shape
    out = torch.zeros(b, rows, columns, dtype=torch.complex128, device="cuda")
    index = []
    for n, m in ((nx, rows), (ny, columns)):
        k = min(n, m)
        low = (k + 1) // 2
        index.append(([*range(low), *range(n - (k - low), n)], [*range(low), *range(m - (k - low), m)]))
    (sx, dx), (sy, dy) = index
    out[:, torch.tensor(dx)[:, None], torch.tensor(dy)[None, :]] = spectra[:, sx][:, :, sy]
    return torch.fft.ifft2(out) * (rows * columns / (nx * ny))


def surrogate_exact(m):
    at, params = 0, []
    for shape in ((103, 16), (64, 18), (64,), (64, 64), (64,), (64, 64), (64,), (1, 64), (1,)):
        n = math.prod(shape)
        params.append(torch.tensor(m["parameters"][at:at + n].reshape(shape), device="cuda", dtype=torch.float64, requires_grad=True))
        at += n
    emb, w1, b1, w2, b2, w3, b3, w4, b4 = params

    def fraction(z, rho, zl, zu):
        z = torch.as_tensor(z.astype(np.int64) - 1, device="cuda")
        rho, zl, zu = (torch.as_tensor(v, device="cuda") for v in (rho, zl, zu))

        def c(edge):
            h = torch.cat([emb[z], ((torch.log(rho) + 1.5) / 2)[:, None], (torch.asinh(edge / rho) / 4)[:, None]], 1)
            for w, b in ((w1, b1), (w2, b2), (w3, b3)):
                h = torch.nn.functional.silu(h @ w.T + b)
            return (h @ w4.T + b4)[:, 0]

        return c(zu) - c(zl)

    loss = ((fraction(*m["batch"]) - torch.as_tensor(m["target"], device="cuda")) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "gradients": np.concatenate([p.grad.cpu().numpy().ravel() for p in params]), "profiles": None}


def exact(case, seed):
    m, kind = model(case, seed), case["kind"]
    if kind in ("scan", "phonons", "waves"):
        return scan_exact(case, m)
    if kind in ("run", "hrtem"):
        field = Field64(case["nx"], case["ny"], m["box"], 200e3)
        ts = list(field.transmissions(m["numbers"], m["positions"], m["dz"], case["slices"]))
        ones = torch.ones(1, case["nx"], case["ny"], dtype=torch.complex128, device="cuda")
        spectrum = field.exits(ones, ts, field.propagator(m["dz"]))[0]
        wave = torch.fft.ifft2(spectrum).cpu().numpy()
        if kind == "run":
            return wave
        alpha = torch.sqrt(field.k2) * field.lam
        slope = 2 * math.pi / field.lam * (m["defocus"] * alpha + 1e7 * alpha ** 3)
        envelope = torch.exp(-(0.05e-3 * slope) ** 2) * torch.exp(-(0.5 * math.pi / field.lam * 30.0 * alpha ** 2) ** 2)
        imaged = torch.fft.ifft2(spectrum * torch.polar(field.soft_aperture(20.0) * envelope, -field.chi(m["defocus"], 1e7)))
        return {"exit": wave, "imaged": imaged.cpu().numpy(), "image": (imaged.abs() ** 2).cpu().numpy()}
    if kind == "jobs":
        out = []
        for j in m["jobs"]:
            field = Field64(j["n"], j["n"], j["box"], j["energy"])
            ts = list(field.transmissions(j["numbers"], j["positions"], j["dz"], j["slices"]))
            if j["at"] is None:
                wave = torch.ones(1, j["n"], j["n"], dtype=torch.complex128, device="cuda")
            else:
                wave = field.probes(20.0, 0.0, 0.0, np.array([j["at"]]))
            out.append((torch.fft.ifft2(field.exits(wave, ts, field.propagator(j["dz"]))[0]).abs() ** 2).cpu().numpy())
        return out
    if kind == "surrogate":
        return surrogate_exact(m)
    v = prepare(case, seed)["values"]
    for axis, step in ((1, 0.25), (0, 0.2)):
        s = case["sigma"] / step
        radius = int(4 * s + 0.5)
        w = [math.exp(-0.5 * x * x / (s * s)) for x in range(-radius, radius + 1)]
        v = sum(wj / sum(w) * torch.roll(v, radius - j, axis) for j, wj in enumerate(w))
    return {"blurred": v, "noisy": None}
