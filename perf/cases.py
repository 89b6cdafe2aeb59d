"""The work a user of this framework has it do, as cases to time: training steps on explicit samples, training of scenes
from rays, rendered frames, and the two network classes on their own, each through its public entry points.

Sizes come from the benchmark's configurations (2^20 samples per step, T = 2^19 and 2^22 tables, 128^3 occupancy grids,
1920x1080 and 1280x720 frames), from NerfOptions' defaults, from the reference benchmark's batch sizes for the network
classes, and, for the small and ragged ones, are generic.

Scene cases do not train a model first: a trained model would differ from run to run.  They write a model that already
knows its scene (`_write_learned_model`): one dense grid level holds the logarithm of the scene's density, the density
network passes it on, everything else is seeded noise of a trained table's size.  Occupancy, sample counts and the
distribution of samples over rays are then those of a scene being trained or rendered."""
import ctypes
import importlib
import math

import numpy as np
import torch

nb = importlib.import_module("3dmaker_b200")
nm = importlib.import_module("3dmaker_b200.nerf")
pl = importlib.import_module("3dmaker_b200.pipeline")
syn = importlib.import_module("3dmaker_b200.synthetic")

LEVELS = 16

# Field samples per ray, counted with these scenes and cameras (800x800 and 1280x720 pictures for training, the orbit's
# frames for rendering, of the large scene those in front of a surface); the pose changes them by a few per cent.
SAMPLES_PER_RAY = {"train": {"sphere": 25.5, "sphere_wide": 8.0, "spheres": 66.0}, "render": {"sphere": 50.0, "spheres": 31.0}}
FIELD_FLOPS = 19456          # density 32-64-16 and colour 32-64-64-8, one sample, forward


def listed():
    return [
        # The benchmark's headline workload: one optimizer step on 2^20 scattered samples, inputs resident.
        {"name": "field_step_1m", "what": "field", "n": 1 << 20, "log2_table": 19, "growth": 1.447},
        # The same step on a handful of samples: fine-tuning on a few rays, where launches and host work count.
        {"name": "field_step_4k", "what": "field", "n": 4096, "log2_table": 19, "growth": 1.447},
        # A batch that fills no tile evenly, on a small table with the default growth factor.
        {"name": "field_step_ragged", "what": "field", "n": 99991, "log2_table": 17, "growth": 1.3819},
        # Samples that a data loader delivers in pinned host memory, copied while the step before runs.
        {"name": "field_step_host", "what": "host", "n": 1 << 18, "log2_table": 19, "growth": 1.447},
        # Training of an object in a box: 65536 rays a call, about seven optimizer steps of 2^18 samples (configuration 3).
        {"name": "train_sphere", "what": "train", "scene": "sphere", "rays": 65536, "log2_table": 19, "color_layers": 3, "priors": False},
        # What a program gets that keeps NerfOptions' defaults (two colour layers, box of +-1), with depth priors; few rays.
        {"name": "train_defaults", "what": "train", "scene": "sphere_wide", "rays": 20011, "log2_table": 19, "color_layers": 2, "priors": True},
        # Training of a large scene: three cascades, a table beyond the cache, 2^21 samples per step (configuration 5).
        {"name": "train_spheres", "what": "train", "scene": "spheres", "rays": 1 << 17, "log2_table": 22, "color_layers": 3, "priors": False},
        # A full frame of a trained object (configuration 4).
        {"name": "render_1080p", "what": "render", "scene": "sphere", "width": 1920, "height": 1080, "log2_table": 19, "rounds": False},
        # A preview while the camera moves: latency.
        {"name": "render_preview", "what": "render", "scene": "sphere", "width": 160, "height": 90, "log2_table": 19, "rounds": False},
        # A frame of the large scene with the option for scenes whose surfaces hide one another.
        {"name": "render_spheres", "what": "render", "scene": "spheres", "width": 1280, "height": 720, "log2_table": 21, "rounds": True},
        # The plain network class on its own: a training step of four layers of 64 (the reference benchmark's batch range).
        {"name": "mlp_step_64x4", "what": "mlp", "n": 1 << 18, "shape": "64-64-64-4"},
        # The grid network class on its own: a training step at the reference benchmark's smallest batch (configuration 1).
        {"name": "grid_step_64k", "what": "grid", "n": 1 << 16, "log2_table": 19, "growth": 1.447, "train": True},
    ]


def _between(rng, lo, hi):
    """A whole number, spread evenly over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


MLP_SHAPES = ("32-64-8-3", "32-64-16-2", "64-64-64-2", "64-64-64-4", "32-32-32-2")


def draw(rng):
    what = rng.choices(("field", "host", "train", "render", "mlp", "grid"), (5, 2, 4, 4, 2, 3))[0]
    growth = rng.choice((1.3819, 1.447))
    if what in ("field", "host"):
        return {"what": what, "n": _between(rng, 1000, 1 << 20), "log2_table": rng.randint(14, 20), "growth": growth}
    if what == "train":
        scene = rng.choice(("sphere", "sphere", "sphere_wide", "spheres"))
        return {"what": what, "scene": scene, "rays": _between(rng, 1000, 1 << 16), "log2_table": rng.randint(17, 21),
                "color_layers": 2 if scene == "sphere_wide" else 3, "priors": rng.random() < 0.3}
    if what == "render":
        scene = rng.choice(("sphere", "sphere", "spheres"))
        width = _between(rng, 64, 1600)
        return {"what": what, "scene": scene, "width": width, "height": max(1, int(width * rng.uniform(0.5, 0.7))),
                "log2_table": rng.randint(17, 21), "rounds": scene == "spheres" and rng.random() < 0.5}
    if what == "mlp":
        return {"what": what, "n": _between(rng, 1000, 1 << 20), "shape": rng.choice(MLP_SHAPES)}
    return {"what": what, "n": _between(rng, 1000, 1 << 20), "log2_table": rng.randint(14, 20), "growth": growth, "train": rng.random() < 0.6}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _network(g, desc):
    """Weights (uniform, +-1/sqrt(inputs)) and small biases of one network, flat."""
    w = [_uniform(g, (o * i,), -i ** -0.5, i ** -0.5) for i, o in desc.layer_dims()]
    return torch.cat(w), _uniform(g, (desc.bias_count,), -0.05, 0.05)


def _moments(g, m, v, scale):
    """Adam moments of a run that has been going on for a while, for gradients of the given size."""
    m.copy_(torch.randn(m.shape, generator=g, device="cuda") * (0.3 * scale))
    v.copy_(_uniform(g, v.shape, 0.5, 1.5) * scale ** 2)


def _samples(g, n):
    """Positions uniform in the unit cube, directions uniform on the sphere, target colours uniform."""
    pos = torch.rand((n, 3), generator=g, device="cuda")
    d = torch.randn((n, 3), generator=g, device="cuda")
    return pos, d / d.norm(dim=1, keepdim=True), torch.rand((n, 3), generator=g, device="cuda").half()


class Fields:
    """A model and its trainer, inputs on the device."""

    def __init__(self, case, seed):
        g = _generator(seed)
        n = case["n"]
        self.model = m = pl.FieldModel(torch, LEVELS, 1 << case["log2_table"], 16, case["growth"])
        m.w[:m.hash_count].copy_(_uniform(g, (m.hash_count,), -0.1, 0.1))
        for off, boff, desc in ((m.off_dw, m.off_db, m.density), (m.off_cw, m.off_cb, m.color)):
            w, b = _network(g, desc)
            m.w[off:off + w.numel()].copy_(w)
            m.w[boff:boff + b.numel()].copy_(b)
        m.w_h.copy_(m.w)
        # gradients are means over the batch: an entry's is about 1 / n of one sample's
        _moments(g, m.m, m.v, 0.1 / n)
        m.step_count = 2000
        self.trainer = pl.SampleTrainer(m, n, lr=1e-3)
        self.n = n
        self.batch = _samples(g, n)

    def state(self):
        m, t = self.model, self.trainer
        return {"loss": t.loss, "colour": t.c_out, "w": m.w, "w_h": m.w_h, "m": m.m, "v": m.v}


class FieldState(Fields):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        pos, dirs, rgb = self.batch
        t = self.trainer
        t.pos[:, :3].copy_(pos)
        t.dirs.copy_(dirs)
        t.target[:, :3].copy_(rgb)

    def run(self):
        self.trainer.step_device(self.n)
        return self.state()


class HostState(Fields):
    """Batches in pinned host memory; the queue is one batch deep, as a loader keeps it."""

    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.batch = [t.cpu().pin_memory() for t in self.batch]
        self.trainer.prefetch(*self.batch)

    def run(self):
        self.trainer.prefetch(*self.batch)
        self.trainer.step_prefetched()
        return self.state()


class _Sphere(syn.SoftSphereScene):
    extent = 0.5


class _WideSphere(syn.SoftSphereScene):
    """The sphere in the default box of +-1."""
    aabb = 1.0
    extent = 1.0


def _scene(case):
    name = case["scene"]
    if name == "sphere":
        return _Sphere(), syn.sphere_cameras(100), (800, 800)
    if name == "sphere_wide":
        return _WideSphere(), syn.sphere_cameras(100, radius=2.0), (800, 800)
    return syn.MultiSphereScene(), syn.sphere_cameras(300, radius=4.5), (1280, 720)


def _options(case):
    o = {"hash_table_size": 1 << case["log2_table"], "color_num_layers": case.get("color_layers", 3), "learning_rate": 1e-3}
    if case["scene"] == "sphere_wide":
        return nm.default_options(**o)
    o.update(aabb_min=(-.5,) * 3, aabb_max=(.5,) * 3, batch_size=1 << 18, render_batch_size=1 << 20, ray_chunk_size=1 << 16, lambda_dist=0.01,
             lambda_depth=0.05 if case.get("priors") else 0.0, beta2=0.99, epsilon=1e-15, loss_scale=128.0)
    if case["scene"] == "spheres":
        o.update(num_cascades=3)
        if case["what"] == "train":
            o.update(batch_size=1 << 21, ray_chunk_size=1 << 17)
    return nm.default_options(**o)


def _world_axis(c, half):
    """Inverse of the contraction, one axis: the unit cube's [0, 1] as [-2, 2], the box as [-1, 1] of that."""
    c = c * 4.0 - 2.0
    far = c.sign() / (2.0 - c.abs()).clamp_min(1e-3)
    return torch.where(c.abs() <= 1.0, c, far) * half


def _write_learned_model(g, eng, scene, opts):
    """Parameters, moments and occupancy of an engine that has been trained on the scene (see the top of the file)."""
    v = eng.arena()
    w = eng.arena_tensor("w")
    T = opts.hash_table_size
    w[:v.sparse_count].copy_(torch.randn((v.sparse_count,), generator=g, device="cuda") * 0.05)
    grid = nb.grid_setup(LEVELS, T, opts.base_resolution, opts.growth_factor)
    level = max(k for k in range(grid.dense_level_start) if grid.scales[k] <= 82.0)
    scale, res = grid.scales[level], int(grid.scales[level]) + 1
    axis = _world_axis(torch.arange(res, device="cuda").float() / scale, float(opts.aabb_max[0]))
    zyx = torch.cartesian_prod(axis, axis, axis)
    log_density = torch.cat([scene.density(torch, p.flip(-1)).clamp_min(1e-4).log() for p in zyx.split(1 << 18)])
    table = w[:v.sparse_count].view(LEVELS, T, 2)
    table[level, :res ** 3, 0] = (log_density + opts.density_bias) / 8.0
    density = nb.mlp_desc(32, opts.density_hidden_dim, 16, opts.density_num_layers)
    color = nb.mlp_desc(32, opts.color_hidden_dim, 8, opts.color_num_layers, 1)
    dw, db = _network(g, density)
    hidden = opts.density_hidden_dim
    first, last = dw[:hidden * 32].view(hidden, 32), dw[-16 * hidden:].view(16, hidden)
    first[:2] = 0.0
    first[0, 2 * level], first[1, 2 * level] = 4.0, -4.0
    last[0] *= 0.05
    last[0, 0], last[0, 1] = 2.0, -2.0
    db[:2] = 0.0
    cw, cb = _network(g, color)
    for t, off in ((dw, v.density_weight_offset), (db, v.density_bias_offset), (cw, v.color_weight_offset), (cb, v.color_bias_offset)):
        w[off:off + t.numel()].copy_(t)
    eng.arena_tensor("w_h").copy_(w)
    eng.occupancy()[1].zero_()
    torch.cuda.synchronize()
    eng.rebuild_occupancy()


class TrainState:
    def __init__(self, case, seed):
        g = _generator(seed)
        scene, poses, (width, height) = _scene(case)
        opts = _options(case)
        self.eng = nm.InstantNerf(torch, opts)
        _write_learned_model(g, self.eng, scene, opts)
        n = case["rays"]
        # the optimizer's second moment as after many steps: the first steps of a fresh optimizer move every parameter by
        # the full learning rate whatever its gradient, which is not the state a program spends its time in
        self.eng.arena_tensor("v").fill_((0.1 / n) ** 2)
        self.o, self.d = syn.random_training_rays(torch, poses, n, width, height, 50.0, seed=int(seed))
        self.rgb = syn.ground_truth(torch, scene, self.o, self.d, (1.0, 1.0, 1.0), extent=scene.extent, steps=96,
                                    chunk=(1 << 14) if case["scene"] == "spheres" else (1 << 17))
        self.out = torch.zeros_like(self.rgb)
        self.depth = self.sigma = None
        if case["priors"]:
            # a third of the rays carry a depth estimate
            some = torch.rand((n,), generator=g, device="cuda") < 1.0 / 3.0
            self.depth = torch.where(some, _uniform(g, (n,), 0.8, 2.2), torch.full((n,), -1.0, device="cuda"))
            self.sigma = _uniform(g, (n,), 0.05, 0.2)
        self.views = {k: self.eng.arena_tensor(k) for k in ("w", "w_h", "m", "v")}
        self.views["bits"], self.views["occupancy"] = self.eng.occupancy()
        for view in self.views.values():
            view.engine = self.eng   # they alias the engine's memory: it lives as long as any of them

    def run(self):
        self.eng.train_rays(self.o, self.d, self.rgb, rgb_out=self.out, depth=self.depth, sigma=self.sigma)
        return dict(self.views, rgb=self.out)


class RenderState:
    """A camera on an orbit around a trained scene: rays from the pose, then the frame."""

    def __init__(self, case, seed):
        g = _generator(seed)
        scene, _, _ = _scene(case)
        opts = _options(case)
        self.eng = nm.InstantNerf(torch, opts, inference=True)
        _write_learned_model(g, self.eng, scene, opts)
        if case["rounds"]:
            self.eng.set_render_rounds(True)
        self.w, self.h = case["width"], case["height"]
        azimuth = float(torch.rand((1,), generator=g, device="cuda").item()) * 360.0
        self.c2w = np.ascontiguousarray(syn.orbit_c2w(azimuth, 20.0, 4.5 if case["scene"] == "spheres" else 1.5), np.float32)
        self.focal = syn.focal_from_fov(self.w, 50.0)
        n = self.w * self.h
        self.o, self.d, self.frame = (torch.zeros((n, 3), device="cuda") for _ in range(3))

    def run(self):
        nb.check(nb.load().nb_generate_rays(self.w, self.h, self.focal, self.c2w.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), 0, self.w * self.h,
                                            nb.ptr(self.o), nb.ptr(self.d), nb.stream_ptr()), "nb_generate_rays")
        self.eng.render(self.o, self.d, self.frame)
        return self.frame


class _Network:
    """A network class's step over the C entry points: the calls in order, with their arguments laid out once."""

    def _adam(self, w, w_h, g, m, v, sparse):
        return self.lib.nb_adam_step, (nb.ptr(w), nb.ptr(w_h), nb.ptr(g), nb.ptr(m), nb.ptr(v), sparse, w.numel(), 1e-3, 0.9, 0.99, 1e-8,
                                       1.0 - 0.9 ** 500, 1.0 - 0.99 ** 500, 1.0 / 128.0, 0, nb.stream_ptr())

    def run(self):
        for fn, args in self.calls:
            nb.check(fn(*args), "network step")
        return self.outputs


def _arena(count):
    return torch.zeros((count + 3) // 4 * 4, device="cuda")


class MlpState(_Network):
    def __init__(self, case, seed):
        gen = _generator(seed)
        self.lib = lib = nb.load()
        n = case["n"]
        k, h, o, layers = (int(x) for x in case["shape"].split("-"))
        self.desc = nb.mlp_desc(k, h, o, layers)
        D = ctypes.byref(self.desc)
        nw = self.desc.weight_count
        w, g, m, v = (_arena(nw + self.desc.bias_count) for _ in range(4))
        weights, biases = _network(gen, self.desc)
        w[:nw].copy_(weights)
        w[nw:nw + biases.numel()].copy_(biases)
        w_h = w.half()
        _moments(gen, m, v, 1e-3)
        x = torch.randn((n, k), generator=gen, device="cuda").half()
        target = torch.rand((n, o), generator=gen, device="cuda").half()
        out = torch.zeros((n, o), device="cuda")
        acts = torch.zeros((max(1, layers - 1), n, h), dtype=torch.float16, device="cuda")
        dloss = torch.zeros((n, o), dtype=torch.float16, device="cuda")
        dx = torch.zeros((n, k), dtype=torch.float16, device="cuda")
        loss = torch.zeros(1, device="cuda")
        P, st = nb.ptr, nb.stream_ptr()
        wb, gb = P(w[nw:]), P(g[nw:])
        self.keep = (x, target, acts, dloss, g)
        self.calls = [(lib.nb_zero_async, (P(g), g.numel() * 4, st)),
                      (lib.nb_mlp_forward, (D, P(x), P(w_h), wb, n, P(out), P(acts), st)),
                      (lib.nb_zero_async, (P(loss), 4, st)),
                      (lib.nb_mse_loss_grad, (P(out), P(target), P(dloss), P(loss), n, o, o, 128.0, 0, st)),
                      (lib.nb_mlp_backward, (D, P(dloss), P(w_h), P(x), P(acts), n, P(g), gb, P(dx), st)),
                      self._adam(w, w_h, g, m, v, 0)]
        self.outputs = {"out": out, "loss": loss, "dx": dx, "w": w, "w_h": w_h, "m": m, "v": v}


class GridState(_Network):
    def __init__(self, case, seed):
        gen = _generator(seed)
        self.lib = lib = nb.load()
        n, T = case["n"], 1 << case["log2_table"]
        self.grid = nb.grid_setup(LEVELS, T, 16, case["growth"])
        self.desc = nb.mlp_desc(2 * LEVELS, 64, 16, 2)
        G, D = ctypes.byref(self.grid), ctypes.byref(self.desc)
        nh, nw, nbias = LEVELS * T * 2, self.desc.weight_count, self.desc.bias_count
        train = case["train"]
        w = _arena(nh + nw + nbias)
        w[:nh].copy_(_uniform(gen, (nh,), -0.1, 0.1))
        weights, biases = _network(gen, self.desc)
        w[nh:nh + nw].copy_(weights)
        w[nh + nw:nh + nw + nbias].copy_(biases)
        w_h = w.half()
        pos = torch.zeros((n, 4), device="cuda")
        pos[:, :3] = torch.rand((n, 3), generator=gen, device="cuda")
        out = torch.zeros((n, 16), device="cuda")
        P, st = nb.ptr, nb.stream_ptr()
        wn_h, wb = P(w_h[nh:]), P(w[nh + nw:])
        self.outputs = {"out": out}
        if not train:
            self.keep = (pos, w, w_h)
            self.calls = [(lib.nb_grid_mlp_forward, (G, D, P(pos), P(w_h), wn_h, wb, n, P(out), None, None, st))]
            return
        g, m, v = (_arena(nh + nw + nbias) for _ in range(3))
        _moments(gen, m, v, 0.1 / n)
        enc, denc = (torch.zeros((n, 2 * LEVELS), dtype=torch.float16, device="cuda") for _ in range(2))
        acts = torch.zeros((n, 64), dtype=torch.float16, device="cuda")
        dloss = torch.zeros((n, 16), dtype=torch.float16, device="cuda")
        target = torch.rand((n, 16), generator=gen, device="cuda").half()
        loss = torch.zeros(1, device="cuda")
        gn, gb = P(g[nh:]), P(g[nh + nw:])
        self.keep = (pos, target, enc, denc, acts, dloss, g)
        self.calls = [(lib.nb_zero_async, (gn, (nw + nbias) * 4, st)),
                      (lib.nb_grid_mlp_forward, (G, D, P(pos), P(w_h), wn_h, wb, n, P(out), P(enc), P(acts), st)),
                      (lib.nb_zero_async, (P(loss), 4, st)),
                      (lib.nb_mse_loss_grad, (P(out), P(target), P(dloss), P(loss), n, 16, 16, 128.0, 0, st)),
                      (lib.nb_mlp_backward, (D, P(dloss), wn_h, P(enc), P(acts), n, gn, gb, P(denc), st)),
                      (lib.nb_hash_scatter_backward, (G, P(pos), P(denc), n, P(g), st)),
                      self._adam(w, w_h, g, m, v, nh)]
        self.outputs.update(loss=loss, w=w, w_h=w_h, m=m, v=v)


STATES = {"field": FieldState, "host": HostState, "train": TrainState, "render": RenderState, "mlp": MlpState, "grid": GridState}


def prepare(case, seed):
    return STATES[case["what"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _touched(case, samples):
    """Entries of the hash table that the corners of so many samples fall on, all levels."""
    T, growth = 1 << case["log2_table"], case.get("growth", 1.3819)
    total = 0.0
    for level in range(LEVELS):
        entries = min(float(T), (16.0 * growth ** level + 1.0) ** 3)
        total += entries * -math.expm1(-8.0 * samples / entries)
    return total


TABLE_READ = 4                      # one entry: two fp16 features
TABLE_UPDATE = 2 * (2 * 4 * 3 + 2)  # ... two parameters with two moments read and written, their fp16 copies written


def work(case):
    what = case["what"]
    if what in ("field", "host"):
        n = case["n"]
        # position, direction, target in; colour row out
        return {"bytes": n * (12 + 12 + 6 + 32) + _touched(case, n) * TABLE_UPDATE, "flops": 3.0 * FIELD_FLOPS * n}
    if what == "train":
        rays = case["rays"]
        samples = rays * SAMPLES_PER_RAY[what][case["scene"]]
        batch = (1 << 21) if case["scene"] == "spheres" else (1 << 18)
        steps = max(1, -(-samples // batch))
        # rays and target colours in, rendered colours out; every optimizer step updates the entries its samples touched
        return {"bytes": rays * (24 + 12 + 12) + steps * _touched(case, samples / steps) * TABLE_UPDATE, "flops": 3.0 * FIELD_FLOPS * samples}
    if what == "render":
        rays = case["width"] * case["height"]
        samples = rays * SAMPLES_PER_RAY[what][case["scene"]]
        return {"bytes": rays * 2 * 12 + rays * 12 + _touched(case, samples) * TABLE_READ, "flops": float(FIELD_FLOPS) * samples}
    n = case["n"]
    if what == "mlp":
        k, h, o, layers = (int(x) for x in case["shape"].split("-"))
        weights = k * h + h * h * (layers - 2) + h * o
        return {"bytes": n * (2 * k + 2 * o + 4 * o + 2 * k) + weights * 26, "flops": 6.0 * weights * n}
    weights = 32 * 64 + 64 * 16
    if case["train"]:
        return {"bytes": n * (12 + 32 + 64) + _touched(case, n) * TABLE_UPDATE, "flops": 6.0 * weights * n}
    return {"bytes": n * (12 + 64) + _touched(case, n) * TABLE_READ, "flops": 2.0 * weights * n}


def tolerance(case):
    # Activations, their gradients and the table are rounded to 16 bits between layers (a relative step of 2^-11), sums are 32
    # bits wide.  Updated parameters carry a small part of that; a parameter whose gradient nearly cancels carries more of it.
    if case["what"] == "train":
        # several optimizer steps in a row, and cells at the occupancy threshold
        return {"rel": 1e-2, "max": 0.5, "differ": 2e-3}
    if case["what"] == "render":
        return {"rel": 2e-3, "max": 0.05}
    return {"rel": 5e-3, "max": 0.5}
