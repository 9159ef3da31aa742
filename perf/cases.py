"""What this library is used for, as calls through its public entry points (slime_b200.capi over the C ABI).

The path is the multi-head Flow-Lenia step and the calls that surround it in a program: a state comes in, it is stepped,
and the state, a field, fitness scalars or logits come out.  It has one direction (the library trains by mutation and
selection, not by gradients) and two data types, fp32 and bf16.  A case names the program:

  forward     a state on the device in, `steps` steps, the normalised state on the device out
  host        the same from and to pinned host memory, copies included
  generation  the reference driver's call for each generation: lift a device field, one step, the channel mean back
  population  independent grids with a weight set for every few of them, `steps` steps, fitness of every grid
  images      host images lifted into grids, `steps` steps, pooled linear read-out to the host
  ring        one torus held as row stripes (here one), halo rows and channel sums exchanged every step

Weights are the seeded draws of slime_b200.inputs in their mass-neutral form, whose trajectories stay finite.  `bell`
puts the state where the growth function bends (0.45 of mass per cell and channel); otherwise every channel has mass 1.
"""
import numpy as np
import torch

from slime_b200 import capi, devmem, inputs

CODE = {"f32": capi.F32, "bf16": capi.BF16}
TORCH = {"f32": torch.float32, "bf16": torch.bfloat16}
# Most cell-updates of a drawn case: bf16 as the largest listed one, fp32 (a slower path) as its own largest.
MOST = {"f32": 64 * 128 * 128 * 4, "bf16": 4096 * 32 * 32 * 24}
IMG = 28                      # edge of an input image; a grid of an `images` case is at least this large


def case(name, do, dtype, batch, height, width, steps, sets=1, bell=False):
    c = {"do": do, "dtype": dtype, "batch": batch, "height": height, "width": width, "steps": steps, "sets": sets, "bell": bell}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest thing a program asks for: one small grid, one step (an interactive view, a unit of a search)
        case("one_step_bf16", "forward", "bf16", 1, 32, 32, 1, bell=True),
        # the reference's own driver: one 128 x 128 grid in fp32, field in and field out, every generation
        case("generation_f32", "generation", "f32", 1, 128, 128, 1, bell=True),
        # the single-organism reference model, fp32 (the repository's first configuration) and its bf16 twin
        case("model_f32", "forward", "f32", 1, 128, 128, 16),
        case("model_bf16", "forward", "bf16", 1, 128, 128, 16),
        # grids that are no multiple of any tile, several weight sets: what users' own field sizes look like
        case("ragged_f32", "forward", "f32", 5, 45, 61, 8, sets=5, bell=True),
        case("ragged_bf16", "forward", "bf16", 6, 75, 53, 8, sets=3, bell=True),
        # the headline: the training-shape batch forward of 64 steps, end to end from host memory
        case("training_bf16", "host", "bf16", 64, 128, 128, 64),
        # the same batch in fp32, the precision the parity runs use; fewer steps, the state stays on the device
        case("training_f32", "forward", "f32", 64, 128, 128, 4),
        # a generation of a population: 16 weight sets x 8 grids, 32 steps, fitness of every grid
        case("population_bf16", "population", "bf16", 128, 128, 128, 32, sets=16),
        # the same in small and in fp32, the size the population parity test runs
        case("population_f32", "population", "f32", 8, 64, 64, 32, sets=4),
        # the supervised-input shape: 4096 images, 24 steps, read-out
        case("images_bf16", "images", "bf16", 4096, 32, 32, 24),
        # one large torus through the row-stripe ring (the large-grid configuration at a quarter of its edge)
        case("torus_bf16", "ring", "bf16", 1, 2048, 2048, 10),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    do = rng.choice(["forward", "forward", "host", "generation", "population", "images", "ring"])
    dtype = rng.choice(["f32", "bf16"])
    steps = 1 if do == "generation" else _log(rng, 2 if do == "population" else 1, {"images": 24, "ring": 16}.get(do, 64))
    most = MOST[dtype] // steps                                   # cells
    if do == "images":
        height, width = rng.randint(IMG, 40), rng.randint(IMG, 40)
    elif do == "ring":
        height, width = _log(rng, 64, 2048), _log(rng, 64, 2048)
    else:
        height, width = _log(rng, 16, 256), _log(rng, 16, 256)
    while height * width > most:
        height, width = max(16, height // 2), max(16, width // 2)
    if do in ("generation", "ring"):
        batch, sets = 1, 1
    elif do == "images":
        batch, sets = _log(rng, 1, min(4096, most // (height * width))), 1
    else:
        per = rng.choice([1, 2, 4, 8])                            # grids that share a weight set
        batch = _log(rng, 1, min(128, max(1, most // (height * width))))
        sets = max(1, min(16, batch // per))
        batch = batch // sets * sets
    return case(None, do, dtype, batch, height, width, steps, sets, rng.random() < 0.5)


def prepare(case, seed):
    c = dict(case)
    B, H, W, dtype = c["batch"], c["height"], c["width"], c["dtype"]
    cells = H * W
    L, Wr, br = inputs.make_lift_readout(seed=seed)
    lifted = c["do"] in ("generation", "images")
    h = capi.Handle(B, H, W, n_weight_sets=c["sets"], dtype=CODE[dtype], stripe=c["do"] == "ring",
                    keep_vprime=c["do"] == "population")
    h.set_weights(inputs.make_weight_sets(c["sets"], seed=seed, bounded=True, mass_profile=L if lifted else None))
    s = {"case": c, "handle": h, "stream": torch.cuda.current_stream().cuda_stream, "L": L, "Wr": Wr, "br": br}
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["do"] == "images":
        rng = np.random.default_rng(seed)
        img = rng.random((B, IMG, IMG), dtype=np.float32)
        s["images"] = np.where(rng.random((B, IMG, IMG), dtype=np.float32) < 0.7, np.float32(0), img)
    elif c["do"] == "generation":
        s["field"] = torch.rand((B, H, W), generator=gen, device="cuda") * (0.9 if c["bell"] else 2.0 / cells)
        s["out"] = torch.empty_like(s["field"])
    else:
        x = torch.rand((B, H, W, 64), generator=gen, device="cuda")
        x *= (0.45 * cells if c["bell"] else 1.0) / x.sum(dim=(1, 2), keepdim=True)
        x = x.to(TORCH[dtype])
        if c["do"] == "host":
            s["x"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
            s["x"].copy_(x)
            s["out"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        else:
            s["x"] = x
            s["out"] = torch.empty_like(x)
        if c["do"] == "ring":
            h.ring_init(None, 0, 1)
    if c["do"] in ("generation", "population", "images"):
        # the state stays in the handle, as in such a program: its buffers, in place (state = stored values x scale)
        stored = devmem.state_view(h)
        scale = devmem.view(h.buffer(capi.BUF_SCALE)[0], (B, 64), torch.float32)
        stored.owner = scale.owner = h            # they live in the handle's memory
        s["state"] = {"stored": stored, "scale": scale}
    return s


def run(s):
    c, h, st = s["case"], s["handle"], s["stream"]
    code, do = CODE[c["dtype"]], c["do"]
    if do == "forward":
        h.set_state_device(s["x"].data_ptr(), code, st)
        h.step(c["steps"], st)
        h.get_state_device(s["out"].data_ptr(), code, st)
        return s["out"]
    if do == "host":
        h.set_state_ptr(s["x"].data_ptr(), code, st)
        h.step(c["steps"], st)
        h.get_state_ptr(s["out"].data_ptr(), code, st)
        return s["out"]
    if do == "ring":
        h.set_state_device(s["x"].data_ptr(), code, st)
        h.ring_sync_mass(st)
        h.step_ring(c["steps"], st)
        h.get_state_device(s["out"].data_ptr(), code, st)
        return s["out"]
    if do == "generation":
        h.lift_field_device(s["field"].data_ptr(), s["L"], st)
        h.step(c["steps"], st)
        h.field_from_state_device(s["out"].data_ptr(), st)
        return {"field": s["out"], "state": s["state"]}
    if do == "images":
        h.lift_images(s["images"], s["L"], st)
        h.step(c["steps"], st)
        return {"logits": h.pool_readout(s["Wr"], s["br"], st), "state": s["state"]}
    h.set_state_device(s["x"].data_ptr(), code, st)
    h.step(c["steps"], st)
    fit = h.fitness(st)
    # hunger is 1 - coherence: its relative error says nothing where the coherence is close to 1
    return {"rank": fit["rank"], "coherence": fit["coherence"], "fitness": fit["fitness"], "state": s["state"]}


def work(case):
    """Bytes: the input, the weights and the result, once each; nothing in between.  Flops: for each cell and step the
    four projections (2 x 64 x 2048), the 3 x 3 stencil (2 x 9 x 512) and the two box sums with what joins them
    (about 24 x 512); for fitness the Gram matrices of the last step (2 x 64 x 512 a cell)."""
    cells = case["batch"] * case["height"] * case["width"]
    e = 2 if case["dtype"] == "bf16" else 4
    n_in = {"images": case["batch"] * IMG * IMG * 4, "generation": cells * 4}.get(case["do"], cells * 64 * e)
    n_out = cells * 64 * e + (cells * 4 if case["do"] == "generation" else 0)
    flops = cells * case["steps"] * (262144 + 2 * 9 * 512 + 24 * 512)
    if case["do"] == "population":
        flops += cells * 2 * 64 * 512
    return {"bytes": n_in + n_out + case["sets"] * 131168 * e, "flops": flops}


def tolerance(case):
    """fp32: sums of 64 to 512 terms in 32 bits, a few dozen steps.  bf16: the state is stored in 8 bits of mantissa after
    every step, which alone costs about 1e-2 over the longer runs."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-2 if case["steps"] <= 8 else 2e-2, "max": 0.4}
