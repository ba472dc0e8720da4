"""Workloads of the framework, each one pass through its public entry points.

Four kinds of work:

* ``operators`` -- the stand-alone SBP operators on (batch, ny, nx) fields: every direction and
  kind that the operator has (diffxi, diffeta and, for the upwind operators, dissxi, disseta).
* ``periodic`` -- euler.System: one periodic curvilinear block, initial vortex, one
  advance_upwind call per step, the field read back to the host, in f64.
* ``blocks`` -- BlockSystem: vortex boundary data on the outer edges, Grid interfaces inside; one
  block, the 2 x 3 multi-block layout, or a batched ensemble of independent instances; from the
  initial vortex over ``steps`` RK4 steps to the packed state on the device.
* ``learned`` -- the learned correction of coarse 64 x 64 states: one Adam step on a batch
  (``train``, returns the updated parameters) or the corrected states (``apply``).

Inputs are drawn from the seed: i.i.d. U[-1, 1) operator fields (the operator configuration of
workloads.py), vortices with the distributions of the batched ensemble, on the repository's
Cartesian and warped grids.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from summationbyparts_b200 import euler, learned, operators, workloads
from summationbyparts_b200.system import BC_GRID, BC_VORTEX, BlockSpec, BlockSystem, Vortice, VortexParameters

OPS = {"upwind4": operators.Upwind4, "upwind9": operators.Upwind9, "sbp8": operators.SBP8}
OP_NAME = {workloads.UPWIND4: "upwind4", workloads.UPWIND9: "upwind9"}
DTYPES = {"f64": torch.float64, "f32": torch.float32}


def listed() -> list[dict]:
    return [
        # one block of the smallest solve's size: four launches, latency
        {"name": "operators_small_f64", "kind": "operators", "op": "upwind4", "dtype": "f64", "batch": 1, "ny": 64,
         "nx": 64},
        # state planes of a block with odd sides, as curvilinear blocks usually have: rows that do
        # not start on 16-byte boundaries
        {"name": "operators_odd_f64", "kind": "operators", "op": "upwind9", "dtype": "f64", "batch": 4, "ny": 1021,
         "nx": 1533},
        {"name": "operators_odd_f32", "kind": "operators", "op": "sbp8", "dtype": "f32", "batch": 4, "ny": 1537,
         "nx": 2047},
        # the operator configuration: 4 fields of 4096 x 4096
        {"name": "operators_field_f64", "kind": "operators", "op": "upwind9", "dtype": "f64", "batch": 4, "ny": 4096,
         "nx": 4096},
        # the smallest solve: one 64 x 64 Cartesian block, vortex boundaries, Upwind4
        {"name": "block64_f64", "kind": "blocks", "layout": "single", "grid": "cartesian", "op": "upwind4",
         "precision": "f64", "ny": 64, "nx": 64, "steps": 20},
        # euler.System of an ordinary size, stepped call by call and read back
        {"name": "periodic_f64", "kind": "periodic", "op": "upwind9", "ny": 193, "nx": 257, "steps": 10},
        # six coupled blocks with uneven sides, in both precisions
        {"name": "multiblock_f64", "kind": "blocks", "layout": "multiblock", "op": "upwind9", "precision": "f64",
         "nx0": 101, "nx1": 81, "ny0": 51, "ny1": 81, "ny2": 73, "steps": 20},
        {"name": "multiblock_f32c", "kind": "blocks", "layout": "multiblock", "op": "upwind9", "precision": "f32c",
         "nx0": 101, "nx1": 81, "ny0": 51, "ny1": 81, "ny2": 73, "steps": 20},
        # the batched ensemble: 512 independent blocks of 48 to 257 points a side, Upwind4 or
        # Upwind9; the compensated form on the tile schedule that the autotuner picks for it
        {"name": "ensemble_f32c", "kind": "blocks", "layout": "ensemble", "precision": "f32c", "instances": 512,
         "stream": 1, "tile_rows": 32, "steps": 3},
        {"name": "ensemble_f64", "kind": "blocks", "layout": "ensemble", "precision": "f64", "instances": 512,
         "stream": 1, "tile_rows": 16, "steps": 3},
        # the learned correction: a training step at its batch size, and a held-out set
        {"name": "correction_train", "kind": "learned", "mode": "train", "batch": 64, "max_batch": 64},
        {"name": "correction_apply", "kind": "learned", "mode": "apply", "batch": 512, "max_batch": 64},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng) -> dict:
    kind = rng.choice(["operators", "operators", "periodic", "single", "multiblock", "ensemble", "learned"])
    op = rng.choice(["upwind4", "upwind9", "sbp8"])
    if kind == "operators":
        ny, nx = _log_int(rng, 32, 4096), _log_int(rng, 32, 4096)
        if rng.random() < 0.5:
            nx -= nx % 4
        return {"kind": "operators", "op": op, "dtype": rng.choice(["f64", "f32"]), "batch": rng.randint(1, 4),
                "ny": ny, "nx": nx}
    if kind == "periodic":
        return {"kind": "periodic", "op": rng.choice(["upwind4", "upwind9"]), "ny": _log_int(rng, 32, 512),
                "nx": _log_int(rng, 32, 512), "steps": 10}
    precision = rng.choice(["f64", "f32c"])
    if kind == "single":
        return {"kind": "blocks", "layout": "single", "grid": rng.choice(["cartesian", "warped"]), "op": op,
                "precision": precision, "ny": _log_int(rng, 32, 1024), "nx": _log_int(rng, 32, 1024), "steps": 10}
    if kind == "multiblock":
        case = {"kind": "blocks", "layout": "multiblock", "op": op, "precision": precision, "steps": 10}
        for side in ("nx0", "nx1", "ny0", "ny1", "ny2"):
            case[side] = _log_int(rng, 32, 192)
        return case
    if kind == "ensemble":
        return {"kind": "blocks", "layout": "ensemble", "precision": precision, "instances": _log_int(rng, 8, 256),
                "stream": rng.randint(2, 1000), "tile_rows": 32 if precision == "f32c" else 16, "steps": 3}
    mode = rng.choice(["train", "apply"])
    return {"kind": "learned", "mode": mode, "batch": _log_int(rng, 4, 64 if mode == "train" else 512),
            "max_batch": 64}


# ----- inputs ------------------------------------------------------------------------------


def _vortex(r, spread: float = 2.0) -> tuple:
    """(x0, y0, eps, mach) with the distributions of the batched ensemble."""
    u = r.random_sample(4)
    return (spread * (2.0 * u[0] - 1.0), spread * (2.0 * u[1] - 1.0), 0.5 + u[2], 0.3 + 0.4 * u[3])


def _params(v) -> VortexParameters:
    return VortexParameters([Vortice(v[0], v[1], workloads.ENSEMBLE_RSTAR, v[2])], mach=v[3])


def _layout(case: dict) -> tuple[list, list]:
    """Blocks of a system case as dicts (x, y, op, bc, instance) and the dt of every instance."""
    outer = [(BC_VORTEX, 0)] * 4
    if case["kind"] == "periodic":
        x, y = workloads.warped(-5.0, 5.0, case["nx"], -5.0, 5.0, case["ny"])
        return [dict(x=x, y=y, op=case["op"], bc=None, instance=0)], [0.2 / (max(case["nx"], case["ny"]) - 1)]
    if case["layout"] == "single":
        make = workloads.cartesian if case["grid"] == "cartesian" else workloads.warped
        x, y = make(-5.0, 5.0, case["nx"], -5.0, 5.0, case["ny"])
        return [dict(x=x, y=y, op=case["op"], bc=outer, instance=0)], [0.2 / (max(case["nx"], case["ny"]) - 1)]
    if case["layout"] == "multiblock":
        specs = workloads.multiblock(OPS[case["op"]](), (case["nx0"], case["nx1"]),
                                     (case["ny0"], case["ny1"], case["ny2"]))
        blocks = [dict(x=s.x, y=s.y, op=case["op"], bc=s.bc, instance=0) for s in specs]
        return blocks, [workloads.multiblock_dt(specs)]
    grids, blocks, dts = {}, [], []
    for i, inst in enumerate(workloads.ensemble_instances(case["instances"], case["stream"])):
        if inst.side not in grids:
            grids[inst.side] = workloads.warped(-5.0, 5.0, inst.side, -5.0, 5.0, inst.side)
        x, y = grids[inst.side]
        blocks.append(dict(x=x, y=y, op=OP_NAME[inst.op_id], bc=outer, instance=i))
        dts.append(inst.dt)
    return blocks, dts


def _vortices(case: dict, seed: int, n: int) -> list:
    r = np.random.RandomState(seed)
    return [_vortex(r, 1.0 if case["kind"] == "periodic" else 2.0) for _ in range(n)]


def _field(case: dict, seed: int) -> torch.Tensor:
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["batch"], case["ny"], case["nx"])
    return torch.rand(shape, dtype=DTYPES[case["dtype"]], device="cuda", generator=g).mul_(2.0).sub_(1.0)


CNN_CIN, CNN_COUT = (16, 32, 32, 32, 32), (32, 32, 32, 32, 8)
CNN_CIN_USED, CNN_COUT_USED = (4, 32, 32, 32, 32), (32, 32, 32, 32, 4)
LEARNING_RATE = 2e-3


def _network(seed: int) -> np.ndarray:
    """Parameters as the library lays them out: per layer weights [cout][9][cin], then biases."""
    r = np.random.RandomState(seed + 1)
    out = []
    for l in range(5):
        w = np.zeros((CNN_COUT[l], 9, CNN_CIN[l]))
        co, ci = CNN_COUT_USED[l], CNN_CIN_USED[l]
        w[:co, :, :ci] = r.standard_normal((co, 9, ci)) * math.sqrt(2.0 / (9 * ci)) * (0.3 if l == 4 else 1.0)
        b = np.zeros(CNN_COUT[l])
        b[:co] = 0.05 * r.standard_normal(co)
        out += [w.ravel(), b]
    return np.concatenate(out).astype(np.float32)


def _pairs(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Coarse states (vortices on the warped 64 x 64 grid) and targets that differ from them by a
    smooth correction of the size that the coarse solve needs."""
    r = np.random.RandomState(seed)
    n = case["batch"]
    v = torch.tensor([_vortex(r) for _ in range(n)], dtype=torch.float64, device="cuda")
    x, y = (torch.from_numpy(a).cuda() for a in workloads.warped(-5.0, 5.0, 64, -5.0, 5.0, 64))
    coarse = _vortex_field(v, x, y, 2.0)
    shifted = v.clone()
    shifted[:, 0] += 2e-3 * torch.from_numpy(r.standard_normal(n)).cuda()
    shifted[:, 1] += 2e-3 * torch.from_numpy(r.standard_normal(n)).cuda()
    return coarse, _vortex_field(shifted, x, y, 2.0)


def _normalisation(coarse, fine_r):
    c = coarse.transpose(0, 1).reshape(4, -1)
    d = (fine_r - coarse).transpose(0, 1).reshape(4, -1)
    return [t.cpu().numpy().astype(np.float32)
            for t in (c.mean(dim=1), c.std(dim=1).clamp_min(1e-6), (d * d).mean(dim=1).sqrt().clamp_min(1e-12))]


def prepare(case: dict, seed: int) -> dict:
    s = {"case": case}
    if case["kind"] == "operators":
        s["prev"] = _field(case, seed)
        op = OPS[case["op"]]()
        s["calls"] = [op.diffxi, op.diffeta] + ([op.dissxi, op.disseta] if op.upwind() is not None else [])
        s["fut"] = [torch.empty_like(s["prev"]) for _ in s["calls"]]
        return s
    if case["kind"] == "learned":
        s["coarse"], s["fine_r"] = _pairs(case, seed)
        net = s["net"] = learned.CorrectionNet(max_batch=case["max_batch"], seed=0)
        net.set_params(_network(seed))
        net.set_normalisation(*_normalisation(s["coarse"], s["fine_r"]))
        return s
    blocks, dts = _layout(case)
    vortices = _vortices(case, seed, len(dts))
    if case["kind"] == "periodic":
        b = blocks[0]
        s["sys"] = euler.System(b["x"], b["y"], OPS[b["op"]]())
        s["vortex"], s["dt"] = _params(vortices[0]), dts[0]
        return s
    specs = [BlockSpec(b["x"], b["y"], OPS[b["op"]](), b["bc"], b["instance"]) for b in blocks]
    system = s["sys"] = BlockSystem(specs, len(dts), case["precision"], 1.4)
    if "tile_rows" in case:
        system.set_tiles(case["tile_rows"], 32)
    for i, v in enumerate(vortices):
        system.set_vortex(_params(v), i)
        system.set_dt(dts[i], i)
    if case["precision"] == "f64":
        s["out"] = torch.empty(system.state_count(0), dtype=torch.float64, device="cuda")
    else:  # hi and lo parts of every block
        s["out"] = torch.empty(system.state_count(1), dtype=torch.float32, device="cuda")
    return s


def run(s: dict):
    case = s["case"]
    if case["kind"] == "operators":
        for call, fut in zip(s["calls"], s["fut"]):
            call(s["prev"], fut)
        return s["fut"]
    if case["kind"] == "learned":
        if case["mode"] == "apply":
            return s["net"].apply(s["coarse"])
        s["net"].train_step(s["coarse"], s["fine_r"], LEARNING_RATE)
        return s["net"].params()
    system = s["sys"]
    if case["kind"] == "periodic":
        system.vortex(0.0, s["vortex"])
        for _ in range(case["steps"]):
            system.advance_upwind(s["dt"])
        return system.field()
    system.init_vortex(0.0)
    system.set_time(0.0)
    system.advance(case["steps"])
    system.get_state_all_device(s["out"].data_ptr(), 0 if case["precision"] == "f64" else 1)
    return s["out"]


# nonzero interior taps of the first derivative and of the dissipation
TAPS = {"upwind4": (6, 7), "upwind9": (10, 11), "sbp8": (8, 0)}


def work(case: dict) -> dict:
    if case["kind"] == "operators":
        n = case["batch"] * case["ny"] * case["nx"]
        size = 8 if case["dtype"] == "f64" else 4
        diff, diss = TAPS[case["op"]]
        # the field is read once; two or four results are written
        return {"bytes": n * size * (5 if diss else 3), "flops": n * 2 * 2 * (diff + diss)}
    if case["kind"] == "learned":
        pixels = case["batch"] * 4096
        flops = 2 * 9 * sum(a * b for a, b in zip(CNN_CIN_USED, CNN_COUT_USED)) * pixels
        if case["mode"] == "train":
            return {"bytes": pixels * 64, "flops": 3 * flops}
        return {"bytes": pixels * 64, "flops": flops}
    # an RK4 step at the least: state and metrics read once, state written once (13 values in f64,
    # 21 with the compensated state's low parts); per stage 4 components x 2 directions of each
    # stencil, the pointwise fluxes and the update
    blocks, _ = _layout(case)
    total = {"bytes": 0, "flops": 0}
    for b in blocks:
        n = b["x"].size * case["steps"]
        diff, diss = TAPS[b["op"]]
        total["bytes"] += n * (21 * 4 if case.get("precision") == "f32c" else 13 * 8)
        total["flops"] += n * 4 * (4 * 2 * 2 * (diff + diss) + 110)
    return total


# ----- the same results from plain torch in 64 bits ------------------------------------------
# Operator coefficients: first boundary weight of H, interior stencils and closure rows of the first
# derivative and of the dissipation (end closures are the flipped start closures, negated for the
# derivative).
TABLES = {
    "upwind4": {
        "h0": 49/144,
        "diff": (
            [-1/24, 1/4, -7/8, 0, 7/8, -1/4, 1/24],
            [
                [-72/49, 187/98, -20/49, -3/98],
                [-187/366, 0, 69/122, -16/183, 2/61],
                [20/123, -69/82, 0, 227/246, -12/41, 2/41],
                [3/298, 16/149, -227/298, 0, 126/149, -36/149, 6/149],
            ],
        ),
        "diss": (
            [1/24, -1/4, 5/8, -5/6, 5/8, -1/4, 1/24],
            [
                [-3/49, 9/49, -9/49, 3/49],
                [3/61, -11/61, 15/61, -9/61, 2/61],
                [-3/41, 15/41, -29/41, 27/41, -12/41, 2/41],
                [3/149, -27/149, 81/149, -117/149, 90/149, -36/149, 6/149],
            ],
        ),
    },
    "upwind9": {
        "h0": 1070017/3628800,
        "diff": (
            [-1/1260, 5/504, -5/84, 5/21, -5/6, 0, 5/6, -5/21, 5/84, -5/504, 1/1260],
            [
                [
                    -1.69567399396458, 2.290233581594, -0.216473500425698, -0.505879766354449,
                    -0.101161106778154, 0.259147072064383, 0.0193922119400659, -0.0495844980755642
                ],
                [
                    -0.442575354959737, 0, 0.191582959381899, 0.282222626681305, 0.112083989713257,
                    -0.151334868892111, -0.0223600502721044, 0.0303806983474913
                ],
                [
                    0.248392603571843, -1.13758367065272, 0, 1.95334726810969, -1.58879011773212,
                    0.393797129320378, 0.252140821030291, -0.121304033647356
                ],
                [
                    0.0829213105268236, -0.239388470313226, -0.27903866639846, 0, 0.343018053395471,
                    0.110370852514749, 0.00172029988649808, -0.0200445645303789, 0.00044118491852249
                ],
                [
                    0.0724159504343116, -0.415199475743626, 0.991181694804303, -1.49802407438608, 0,
                    1.30188867830442, -0.603535071819214, 0.173429775718218, -0.0240842144699299,
                    0.00192673715759439
                ],
                [
                    -0.0597470838462221, 0.180551858630298, -0.0791241454636765, -0.155240829877729,
                    -0.419298775383066, 0, 0.642287612546289, -0.148833147569152, 0.046540760980226,
                    -0.00775679349670433, 0.000620543479736347
                ],
                [
                    -0.00619425252179959, 0.0369595678895333, -0.0701892820620398, -0.00335233082197107,
                    0.269304373763091, -0.889857974743355, 0, 0.86665664552233, -0.257919763669076,
                    0.064479940917269, -0.0107466568195448, 0.000859732545563586
                ],
                [
                    0.014485349101433, -0.0459275574977554, 0.0308833474560615, 0.0357240610228828,
                    -0.0707760049349999, 0.188587240076292, -0.792626447113877, 0, 0.825608497215073,
                    -0.235888142061449, 0.0589720355153623, -0.00982867258589373, 0.000786293806871498
                ],
            ],
        ),
        "diss": (
            [1/1260, -1/126, 1/28, -2/21, 1/6, -1/5, 1/6, -2/21, 1/28, -1/126, 1/1260],
            [
                [
                    -0.000399020778658945, 0.00205394169917502, -0.00424493243399805, 0.00438126393542801,
                    -0.00218883813216888, 0.000298565988131608, 0.000138484104084115, -3.94643819928825e-05
                ],
                [
                    0.000396913216138553, -0.00228230530115522, 0.00543069719436758, -0.00681086901935894,
                    0.00469064759201504, -0.00161429862514855, 0.000162083873811316, 2.71310693302277e-05
                ],
                [
                    -0.00487084939816571, 0.0322464611075207, -0.0906094757860846, 0.139830191253413,
                    -0.127675500367419, 0.0687310321912961, -0.020091770221527, 0.00243991122096699
                ],
                [
                    0.000718155125886276, -0.00577715378536685, 0.0199749582302141, -0.0387940986951101,
                    0.0462756436981388, -0.0346770570075288, 0.0159058082995305, -0.00406744078428648,
                    0.00044118491852249
                ],
                [
                    -0.00156687484682703, 0.0173758484693946, -0.0796515646886111, 0.202094401829054,
                    -0.316098733124618, 0.31799924013125, -0.20652292891114, 0.083711245559847,
                    -0.0192673715759439, 0.00192673715759439
                ],
                [
                    6.88352254356072e-05, -0.00192595810396278, 0.0138098624496279, -0.0487746083763075,
                    0.102417890394006, -0.13829222666962, 0.123829022892659, -0.0734723830823462,
                    0.0279244565881356, -0.00620543479736347, 0.000620543479736347
                ],
                [
                    4.4234536710064e-05, 0.000267913080025652, -0.00559301314813691, 0.0309954862110834,
                    -0.0921529346596015, 0.171559035817103, -0.212738289547735, 0.179835101537893,
                    -0.10316790546763, 0.0386879645503614, -0.00859732545563586, 0.000859732545563586
                ],
                [
                    -1.15289127131636e-05, 4.10149803795578e-05, 0.000621188131452618, -0.00724912245235322,
                    0.0341622279353287, -0.0930972311856124, 0.164473506705108, -0.198013074867399,
                    0.165121699443015, -0.0943552568245798, 0.0353832213092174, -0.00786293806871498,
                    0.000786293806871498
                ],
            ],
        ),
    },
    "sbp8": {
        "h0": 0.294890676177879,
        "diff": (
            [
                0.00357142857142857, -0.0380952380952381, 0.2, -0.8, 0, 0.8, -0.2, 0.0380952380952381,
                -0.00357142857142857
            ],
            [
                [
                    -1.6955436044319, 2.24741246341404, -0.03389319226015, -0.781028168126749,
                    0.0254881486107905, 0.343865227388873, -0.0862858162633335, -0.0200150583315761
                ],
                [
                    -0.434378988266985, 0, 0.0918511925072956, 0.494008626807984, -0.0246151762937235,
                    -0.186759403432935, 0.0527267838475813, 0.00716696483080115
                ],
                [
                    0.0388218088704253, -0.544329744454984, 0, 0.389516189693211, 0.136433486528546,
                    0.103290582800845, -0.179720579323281, 0.0559882558852296
                ],
                [
                    0.128088632226564, -0.419172130036008, -0.0557707021445779, 0, 0.124714160903055,
                    0.2812852125191, -0.0394470423942641, -0.019698131073843
                ],
                [
                    -0.0182119472519009, 0.090998664615455, -0.0851090570277506, -0.543362886365301, 0,
                    0.637392455438558, -0.102950081118829, 0.0298964956216039, -0.0086536439119011
                ],
                [
                    -0.0793147196245203, 0.222875323171502, -0.0207999824391436, -0.395611167748401,
                    -0.205756876210586, 0, 0.545876519966127, -0.0942727926638298, 0.029797181295285,
                    -0.00279348574643297
                ],
                [
                    0.0275587615266177, -0.0871295642560637, 0.0501135077563584, 0.0768229253600969,
                    0.0460181213406519, -0.75587358166358, 0, 0.821713248844682, -0.216615355227872,
                    0.0412600676624518, -0.00386813134335486
                ],
                [
                    0.00584767272160451, -0.0108336661209337, -0.0142810403117803, 0.0350919361287023,
                    -0.0122244235731112, 0.119411743193552, -0.751668243727123, 0, 0.792601963555477,
                    -0.198150490888869, 0.0377429506454989, -0.00353840162301552
                ],
            ],
        ),
    },
}


def _matrix(op: str, kind: str, n: int) -> torch.Tensor:
    diag, start = TABLES[op][kind]
    d = np.zeros((n, n))
    h = len(diag) // 2
    for k, c in enumerate(diag):
        i = np.arange(len(start), n - len(start))
        d[i, i + k - h] = c
    sign = -1.0 if kind == "diff" else 1.0
    for i, row in enumerate(start):
        for k, c in enumerate(row):
            d[i, k] = c
            d[n - 1 - i, n - 1 - k] = sign * c
    return torch.from_numpy(d * (n - 1)).cuda()


def _vortex_field(v, x, y, t):
    """(n, 4, ny, nx) of the vortices v[n] = (x0, y0, eps, mach) at time t, radius 1, gamma 1.4."""
    x0, y0, eps, mach = (v[:, k, None, None] for k in range(4))
    p_inf = 1.0 / (1.4 * mach * mach)
    dx, dy = x - x0 - t, y - y0
    f = 1.0 - (dx * dx + dy * dy)
    rho = (1.0 - eps ** 2 * 0.4 * mach ** 2 / (8.0 * math.pi ** 2 * p_inf) * torch.exp(f)) ** 2.5
    w = eps / (2.0 * math.pi * torch.sqrt(p_inf)) * torch.exp(f / 2.0)
    u, vv, p = 1.0 - w * dy, w * dx, rho ** 1.4 * p_inf
    return torch.stack([rho, rho * u, rho * vv, p / 0.4 + rho * (u * u + vv * vv) / 2.0], dim=1)


class _Block:
    def __init__(self, b: dict, cache: dict):
        self.bc, self.instance = b["bc"], b["instance"]
        self.x, self.y = torch.from_numpy(b["x"]).cuda(), torch.from_numpy(b["y"]).cuda()
        ny, nx = self.x.shape

        def mat(kind, n):
            key = (b["op"], kind, n)
            if key not in cache:
                cache[key] = _matrix(*key)
            return cache[key]

        self.dx, self.dy = mat("diff", nx).T, mat("diff", ny)
        self.upwind = "diss" in TABLES[b["op"]]
        if self.upwind:
            self.sx, self.sy = mat("diss", nx).T, mat("diss", ny)
        x_xi, x_eta = self.x @ self.dx, self.dy @ self.x
        y_xi, y_eta = self.y @ self.dx, self.dy @ self.y
        self.det = x_xi * y_eta - x_eta * y_xi
        self.xi, self.eta = (y_eta, -x_eta), (-y_xi, x_xi)
        self.hi = ((nx - 1) / TABLES[b["op"]]["h0"], (ny - 1) / TABLES[b["op"]]["h0"])

    def rhs(self, q):
        rho, mu, mv, e = q
        u, v = mu / rho, mv / rho
        p = 0.4 * (e - 0.5 * (mu * u + mv * v))
        ef = torch.stack([mu, mu * u + p, mu * v, u * (e + p)])
        ff = torch.stack([mv, mv * u, mv * v + p, v * (e + p)])
        k = -((self.xi[0] * ef + self.xi[1] * ff) @ self.dx) - self.dy @ (self.eta[0] * ef + self.eta[1] * ff)
        if self.upwind:
            c = torch.sqrt(1.4 * p / rho)
            for m, left in ((self.xi, False), (self.eta, True)):
                a = (torch.abs(m[0] * u + m[1] * v) + c * torch.sqrt(m[0] ** 2 + m[1] ** 2)) * q
                k = k + (self.sy @ a if left else a @ self.sx)
        return k / self.det

    # sides: (edge index, sign, tau, metric pair, hi)
    SIDES = ((("row", -1), -1.0, 1.0, "eta", 1), (("row", 0), 1.0, -1.0, "eta", 1),
             (("col", -1), -1.0, 1.0, "xi", 0), (("col", 0), 1.0, -1.0, "xi", 0))

    @staticmethod
    def edge(a, where):
        return a[..., where[1], :] if where[0] == "row" else a[..., :, where[1]]

    def sat(self, q, k, side, z):
        where, sign, tau, m, h = self.SIDES[side]
        y = self.edge(q, where)
        det = self.edge(self.det, where)
        kx_, ky_ = (self.edge(c, where) / det for c in getattr(self, m))
        r = torch.sqrt(kx_ ** 2 + ky_ ** 2)
        kx, ky = kx_ / r, ky_ / r
        rho, u, v = y[0], y[1] / y[0], y[2] / y[0]
        p = 0.4 * (y[3] - 0.5 * rho * (u * u + v * v))
        c = torch.sqrt(1.4 * p / rho)
        th, phi2, al, be = kx * u + ky * v, 0.2 * (u * u + v * v), rho / (math.sqrt(2.0) * c), 1.0 / (2.0 * c * c)
        g, d, w = (phi2 + c * c) / 0.4, y - z, ky * u - kx * v
        cu = kx_ * u + ky_ * v
        t = ((1 - phi2 / c ** 2) * d[0] + 0.4 / c ** 2 * (u * d[1] + v * d[2] - d[3]),
             (-w * d[0] + ky * d[1] - kx * d[2]) / rho,
             be * ((phi2 - c * th) * d[0] + (kx * c - 0.4 * u) * d[1] + (ky * c - 0.4 * v) * d[2] + 0.4 * d[3]),
             be * ((phi2 + c * th) * d[0] - (kx * c + 0.4 * u) * d[1] - (ky * c + 0.4 * v) * d[2] + 0.4 * d[3]))
        l0, l1, l2, l3 = ((s + sign * torch.abs(s)) * a for s, a in zip((cu, cu, cu + c * r, cu - c * r), t))
        out = torch.stack([l0 + al * (l2 + l3),
                           u * l0 + ky * l1 + al * ((u + kx * c) * l2 + (u - kx * c) * l3),
                           v * l0 - kx * l1 + al * ((v + ky * c) * l2 + (v - ky * c) * l3),
                           phi2 / 0.4 * l0 + rho * w * l1 + al * ((g + c * th) * l2 + (g - c * th) * l3)])
        self.edge(k, where).add_(out * (self.hi[h] * tau))


def _exact_steps(case: dict, seed: int) -> list:
    """The state (4, ny, nx) of every block after the case's steps."""
    specs, dts = _layout(case)
    cache = {}
    blocks = [_Block(b, cache) for b in specs]
    vor = torch.tensor(_vortices(case, seed, len(dts)), dtype=torch.float64, device="cuda")
    opposite = (1, 0, 3, 2)

    def vortex(b, x, y, t):
        return _vortex_field(vor[b.instance:b.instance + 1], x, y, t)[0]

    def rhs_all(qs, c):
        out = []
        for b, q in zip(blocks, qs):
            k = b.rhs(q)
            for side in range(4):
                where = b.SIDES[side][0]
                if b.bc is None:
                    z = b.edge(q, b.SIDES[opposite[side]][0])
                elif b.bc[side][0] == BC_GRID:
                    z = b.edge(qs[b.bc[side][1]], b.SIDES[opposite[side]][0])
                else:
                    x, y = (b.edge(a, where)[None, :] for a in (b.x, b.y))
                    z = vortex(b, x, y, time[b.instance] + c * dts[b.instance])[:, 0]
                b.sat(q, k, side, z)
            out.append(k)
        return out

    time = [0.0] * len(dts)
    qs = [vortex(b, b.x, b.y, 0.0) for b in blocks]
    dt = [dts[b.instance] for b in blocks]
    for _ in range(case["steps"]):
        acc, u = qs, qs
        for a, w, c in ((0.5, 1 / 6, 0.0), (0.5, 1 / 3, 0.5), (1.0, 1 / 3, 0.5), (None, 1 / 6, 1.0)):
            k = rhs_all(u, c)
            acc = [q + w * h * kk for q, h, kk in zip(acc, dt, k)]
            if a is not None:
                u = [q + a * h * kk for q, h, kk in zip(qs, dt, k)]
        qs = acc
        time = [t + h for t, h in zip(time, dts)]
    return qs


def _net(params, coarse, mean, scale):
    """Network output (n, 4, 64, 64) in the precision of its arguments."""
    a, off = (coarse - mean[:, None, None]) / scale[:, None, None], 0
    for l in range(5):
        ci, co = CNN_CIN[l], CNN_COUT[l]
        w = params[off:off + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        b = params[off + co * 9 * ci:off + co * 9 * ci + co]
        off += co * 9 * ci + co
        w, b = w[:CNN_COUT_USED[l], :CNN_CIN_USED[l]], b[:CNN_COUT_USED[l]]
        # a 3x3 convolution as nine products
        ap = torch.nn.functional.pad(a, (1, 1, 1, 1))
        a = b[None, :, None, None] + sum(
            torch.einsum("nchw,oc->nohw", ap[:, :, dy:dy + 64, dx:dx + 64], w[:, :, dy, dx])
            for dy in range(3) for dx in range(3))
        if l < 4:
            a = torch.nn.functional.gelu(a)
    return a


def exact(case: dict, seed: int):
    if case["kind"] == "operators":
        prev = _field(case, seed).double()
        kinds = ("diff", "diss") if "diss" in TABLES[case["op"]] else ("diff",)
        out = []
        for kind in kinds:
            out += [prev @ _matrix(case["op"], kind, case["nx"]).T, _matrix(case["op"], kind, case["ny"]) @ prev]
        return out
    if case["kind"] == "learned":
        coarse, fine_r = _pairs(case, seed)
        mean, scale, oscale = (torch.from_numpy(a).double().cuda() for a in _normalisation(coarse, fine_r))
        params = torch.from_numpy(_network(seed)).double().cuda()
        if case["mode"] == "apply":
            return torch.cat([c + _net(params, c, mean, scale) * oscale[:, None, None] for c in coarse.split(64)])
        params.requires_grad_(True)
        y = _net(params, coarse, mean, scale)
        ((y - (fine_r - coarse) / oscale[:, None, None]) ** 2).mean().backward()
        g = params.grad  # the first Adam step: the bias corrections cancel the moments' factors
        return (params - LEARNING_RATE * g / (torch.sqrt(g * g) + 1e-8)).detach().cpu().numpy()
    qs = _exact_steps(case, seed)
    if case["kind"] == "periodic":
        return qs[0].cpu().numpy()
    if case["precision"] == "f64":
        return torch.cat([q.reshape(-1) for q in qs])
    parts = []
    for q in qs:  # hi then lo planes of every block
        hi = q.float().double()
        parts += [hi.reshape(-1), (q - hi).reshape(-1)]
    return torch.cat(parts)
