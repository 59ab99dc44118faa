"""Workloads of the collapse integrator, through the calls a user's program makes.

A user of this package integrates the chemistry of a grid of cells: in one call
from a state to the end of its collapse (``run_cells``, ``Context.run``; several
sub-grids batched, or one of the other outer-step policies), step by step beside
their own hydrodynamics (``Context.upload`` / ``prepare`` / ``advance`` /
``download``), on records that stay in their own device buffer
(``wr_advance_cells_noalloc``), or with gradients (``diff.collapse_chemistry``).
A case is one of these on a grid of given size and stage of the collapse.

The grids are those of the reference's own collapse: ``STAGES`` holds the
reference cell's state after so many outer steps (density from 1e-23 to 1e-6 g/cm3),
and every cell of a grid is that state with its density scaled by a seeded factor
in [0.8, 1.2], the reference's perturbation.  The stages differ in stiffness: 6
to 60 ROS2S attempts per cell and outer step.

No output has a value that plain numpy gives in seconds: each is the end of an
adaptive integration through the whole network, so ``exact`` has none.
"""
import ctypes

import numpy as np
import torch

import warp_reactor_gb300 as wr
from warp_reactor_gb300 import diff

# outer step: (ROS2S attempts per cell and outer step there, rho, T, e, density driver,
# the 14 number densities)
STAGES = {
    25: (5.9, 2.3753340362823066e-23, 534.153848955889, 54769729954.26469, 2.3753340362823083e-23,
          (0.00025618552549788937, 0.00025618556150480427, 10.83404713075661, 3.6640273862995257e-11, 1e-100, 1e-100, 6.333589729817888e-13,
           1.6881562241392876e-28, 0.0007538835192845933, 4.6867915540768345e-30, 1e-100, 7.29240346788168e-43, 4.178169560203495e-43, 0.8396897106125968)),
    125: (7.7, 3.2733557531591786e-19, 385.22426801321996, 39492983765.66005, 3.273355753159182e-19,
          (0.03142915467127691, 0.03142915765474051, 149173.31096206798, 3.025094550689668e-09, 1.14751673366209e-19, 6.242907888942967e-13, 4.163094616247876e-11,
           1.6107830949101412e-26, 75.38476829084823, 3.5337428341617813e-28, 7.054248196868684e-16, 3.1011456170695158e-49, 9.027268669248522e-52, 11571.43838768974)),
    225: (10.1, 4.51088466846136e-15, 895.012378831429, 91676232862.19997, 4.5108846684613635e-15,
          (6.583491949036527, 6.583493683094265, 2044112304.913061, 1.7782040920124798e-06, 2.5811147789880335e-17, 8.541808144249525e-09, 4.414635335692567e-08,
           8.41506834438941e-24, 6832693.984417485, 3.331693972769552e-25, 7.273972504799058e-11, 1.866424755968225e-54, 7.367121109375478e-59, 159461506.63488907)),
    275: (33.8, 5.295365984726208e-13, 1035.3502084208274, 94757586052.29124, 5.29536598472621e-13,
          (79.02607613218615, 79.02610086364804, 73823965507.44606, 2.5473655395079392e-05, 2.829541388109127e-16, 2.752035500208194e-07, 7.421934865506078e-07,
           1e-100, 83870156795.29376, 4.662580672847096e-24, 8.24242237310555e-07, 1.7841997804126058e-57, 2.7883569413770916e-49, 18719322265.350815)),
    325: (9.2, 6.216275292571373e-11, 1519.2279233846252, 131786981617.61998, 6.216275292571375e-11,
          (918.3929260705307, 918.3588355783321, 126538490116.05998, 0.00046724222925079563, 3.4042767576275296e-15, 3.2707411536043023e-07, 0.03455773442780189,
           1.3013642887030917e-21, 14115449133414.68, 9.123575000332881e-23, 0.0001225121139894861, 2.579225015637234e-60, 1.6358457293777322e-29, 2197477206059.4072)),
    375: (33.5, 7.297338583299314e-09, 2076.908405567025, 181931913270.02426, 7.297338583299315e-09,
          (6649.281648793222, 6648.480184413076, 193563962495938.97, 0.008949976569956913, 2.4546564264538983e-14, 0.00043199480403778974, 0.8104143567160758,
           1.982492256485715e-20, 1567669861992514.2, 1.06561298234639e-21, 0.013958043870070004, 1.8410812161805048e-61, 4.0688065885230125e-20, 257963723403014.88)),
    400: (45.0, 7.906451771939037e-08, 2150.591012901076, 187254240056.34845, 7.906451771939041e-08,
          (9377.70765070346, 9373.817184252604, 900109664672593.0, 0.036006325557116886, 3.626745062959504e-14, 0.0019312001134954358, 3.926472776413871,
           1.0000000000000075e-100, 1.7583791446136858e+16, 1.0000000000000076e-100, 0.15285260267677617, 2.9495808168870188e-61, 1.0579846927659922e-18, 2794961087133032.0)),
    425: (58.4, 8.566408000454138e-07, 2802.7060842521396, 249237817797.6299, 8.566408000454144e-07,
          (17371.31038907167, 17360.63137075347, 5.549514398701912e+16, 0.7614755576596474, 1.0000000001406804e-100, 0.11242368605740981, 11.440493875861788,
           1.0000000001406805e-100, 1.6764384944645658e+17, 1.0000000001406805e-100, 1.520105560150084, 1.4474324799407755e-60, 2.585823917486757e-13, 3.028258151010253e+16)),
    430: (64.5, 1.3796285748811394e-06, 2943.5876499337924, 263222572040.6166, 1.3796285748811402e-06,
          (19019.869918698776, 19006.911558657648, 1.0901016139283784e+17, 1.3049952333306678, 1.0000000000000003e-100, 0.2241722305498497, 14.263355274450927,
           1.0000000000000001e-100, 2.6017475743326022e+17, 1.0000000000000003e-100, 2.431822093046285, 2.114200501138369e-60, 1.9498176474553207e-12, 4.877040035463988e+16)),}
# operations of one ROS2S attempt: the fused Jacobian and RHS, two RHS evaluations
# (an exp or log counted as 20), the 15x15 factorisation, three solves, the combinations
ATTEMPT_FLOPS = 26000
# outer steps from a stage to the end of the collapse, and attempts per cell over them
TO_THE_END = {400: (45, 2300), 425: (13, 800), 430: (8, 500)}
MATH = {"cuda": wr.MATH_CUDA, "portable": wr.MATH_PORTABLE}
POLICY = {"independent": wr.POLICY_GRIDWIDE_INDEPENDENT, "legacy": wr.POLICY_LEGACY_LOCAL,
          "cta32": wr.POLICY_GRIDWIDE_CTA32}


def listed():
    return [
        # the single-cell program, the last tenth of its collapse: one cell, one stream of steps
        {"name": "run 1 cell", "do": "run", "grids": "1", "stage": 400, "policy": "independent", "math": "cuda",
         "perturb": False},
        # the structured policy's controller per tile of 32 cells, a grid with a ragged last tile
        {"name": "run 1000 cells cta32", "do": "run", "grids": "1000", "stage": 430, "policy": "cta32",
         "math": "cuda", "perturb": True},
        # the batching form: sub-grids of several sizes in one context, to the end of the collapse
        {"name": "run 4 grids", "do": "run", "grids": "512,1000,216,64", "stage": 425, "policy": "independent",
         "math": "cuda", "perturb": True},
        # the smallest coupled call: a 2^3 grid, one outer step
        {"name": "step 2^3", "do": "step", "cells": 8, "stage": 25, "steps": 1, "math": "cuda"},
        # a small grid coupled step by step
        {"name": "step 8^3", "do": "step", "cells": 512, "stage": 325, "steps": 3, "math": "cuda"},
        # the size of the gradient workload and of most checks, at a stiff stage
        {"name": "step 16^3", "do": "step", "cells": 4096, "stage": 375, "steps": 2, "math": "cuda"},
        # a block of cells of no round size, in the arithmetic the CPU oracle reproduces
        {"name": "step 20011 portable", "do": "step", "cells": 20011, "stage": 225, "steps": 2, "math": "portable"},
        # 32^3 in the middle of the H2-forming phase, the stiffest part before the end
        {"name": "step 32^3", "do": "step", "cells": 32768, "stage": 275, "steps": 1, "math": "cuda"},
        # the benchmark's 64^3 grid
        {"name": "step 64^3", "do": "step", "cells": 262144, "stage": 125, "steps": 2, "math": "cuda"},
        # gradients of the 16^3 differentiation workload over a few outer steps
        {"name": "diff 16^3", "do": "diff", "cells": 4096, "stage": 125, "steps": 4},
        # gradients of a small sample of cells over a longer stretch
        {"name": "diff 64 cells", "do": "diff", "cells": 64, "stage": 325, "steps": 8},
        # a caller that cannot allocate device memory, its records in its own buffer
        {"name": "noalloc 1000", "do": "noalloc", "cells": 1000, "stage": 225},
    ]


def _log_int(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def draw(rng):
    do = rng.choice(["run", "step", "step", "step", "diff", "noalloc"])
    stage = rng.choice(sorted(STAGES))
    if do == "step":
        steps = rng.randint(1, 3)
        most = min(262144, 262144 * 2 * 7.7 / (STAGES[stage][0] * steps))
        return {"do": do, "cells": _log_int(rng, 1, most), "stage": stage, "steps": steps,
                "math": rng.choice(["cuda", "cuda", "cuda", "portable"])}
    if do == "diff":
        return {"do": do, "cells": _log_int(rng, 1, 4096), "stage": stage,
                "steps": rng.randint(1, max(1, int(100 / STAGES[stage][0])))}
    if do == "noalloc":
        return {"do": do, "cells": _log_int(rng, 1, 4096), "stage": stage}
    policy = rng.choice(["independent", "independent", "legacy", "cta32"])
    if policy == "independent" and rng.random() < 0.5:
        grids = [_log_int(rng, 1, 1000) for _ in range(rng.randint(2, 6))]
    else:
        grids = [_log_int(rng, 1, 1000 if policy == "cta32" else 3000)]
    return {"do": do, "grids": ",".join(map(str, grids)), "stage": 430 if policy == "cta32" else 425, "policy": policy,
            "math": rng.choice(["cuda", "cuda", "cuda", "portable"]), "perturb": rng.random() < 0.75}


def _grid(cells, stage, rng):
    _, rho, T, e, driver, xn = STAGES[stage]
    c = np.zeros(cells, wr.COLLAPSE_STATE)
    f = rng.uniform(0.8, 1.2, cells)
    c["rho"], c["T"], c["e"], c["density_driver"] = rho * f, T, e, driver * f
    c["xn"] = np.array(xn)[None, :] * f[:, None]
    return c


def _sizes(case):
    return [int(g) for g in str(case.get("grids", case.get("cells"))).split(",")]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    cells = np.concatenate([_grid(n, case["stage"], rng) for n in _sizes(case)])
    s = {"case": case, "cells": cells}
    if case["do"] == "run":
        s["context"] = wr.Context(grids=_sizes(case), math=MATH[case["math"]])
        s["context"].set_policy(POLICY[case["policy"]])
        s["out"] = np.empty_like(cells)
    elif case["do"] == "step":
        s["context"] = wr.Context(len(cells), math=MATH[case["math"]])
        s["out"] = np.empty_like(cells)
    elif case["do"] == "noalloc":
        with wr.Context(len(cells), math=wr.MATH_PORTABLE) as ctx:
            ctx.upload(cells)
            s["dt"] = ctx.prepare(0, 0.0, 0, False)[1]
        s["records"] = torch.from_numpy(cells.view(np.uint8)).cuda()
        s["advance"] = wr.lib().wr_advance_cells_noalloc
        s["advance"].argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double,
                                 ctypes.POINTER(ctypes.c_int)]
    else:
        # the grid timesteps of a plain run of the grid, as diff.schedule takes them, for the first outer steps
        time, dts = 0.0, []
        with wr.Context(len(cells), math=wr.MATH_PORTABLE) as ctx:
            ctx.upload(cells)
            for step in range(case["steps"]):
                _, dt = ctx.prepare(step, time, step, True)
                ctx.advance(step, time + dt, dt)
                time += dt
                dts.append(dt)
        s["schedule"] = np.array(dts)
        s["map"] = diff.DiffMap(len(cells), max_outer_steps=case["steps"], max_accepted_per_cell=4096)
        s["records"] = torch.from_numpy(cells.view(np.uint8)).cuda()
        s["u"] = torch.from_numpy(diff.initial_u(cells)).cuda().requires_grad_()
        # multipliers of a fit while the gas is thin; at the network's own rates in the dense gas, where scaled
        # rates beside the network's own Jacobian take the integrator thousands of steps
        p = rng.normal(0.0, 0.01, diff.num_multipliers()) * (1.0 if case["stage"] <= 125 else 0.0)
        s["p"] = torch.from_numpy(p).cuda().requires_grad_()
        # the loss weights the final abundances and temperature by their sizes
        _, _, T, _, _, xn = STAGES[case["stage"]]
        s["scale"] = torch.tensor([max(x, 1e-20) for x in xn] + [T], dtype=torch.float64, device="cuda")
    return s


def _fields(cells):
    words = cells.view(np.int64).reshape(len(cells), 27)
    out = {k: cells[k] for k in ("rho", "T", "e", "xn", "time", "density_driver", "completed_steps")}
    out["stats"] = words[:, 20:]
    return out


def run(s):
    case = s["case"]
    if case["do"] == "run":
        ctx, out = s["context"], s["out"]
        ctx.upload(s["cells"])
        result, steps = ctx.run(case["perturb"])
        ctx.download(out)
        return {"result": result, "steps": steps, "cells": _fields(out)}
    if case["do"] == "step":
        # a block of outer steps from step 20 on, the first of which perturbs the grid
        ctx, out, time, done = s["context"], s["out"], 0.0, []
        ctx.upload(s["cells"])
        for step in range(case["steps"]):
            result, dt = ctx.prepare(step, time, 20 + step, True)
            result2, cells = ctx.advance(step, time + dt, dt)
            time += dt
            done += [result, result2, cells]
        ctx.download(out)
        return {"done": done, "time": time, "cells": _fields(out)}
    if case["do"] == "noalloc":
        records, n = s["records"].clone(), ctypes.c_int()
        result = s["advance"](records.data_ptr(), len(s["cells"]), 0, s["dt"], s["dt"], ctypes.byref(n))
        return {"result": result, "cells": n.value,
                "state": records.view(torch.float64).view(-1, 27)[:, :19],
                "counts": records.view(torch.int64).view(-1, 27)[:, 19:]}
    s["u"].grad = s["p"].grad = None
    q = diff.collapse_chemistry(s["u"], s["p"], s["map"], s["records"], s["schedule"], True)
    (q / s["scale"]).square().sum().backward()
    return {"q": q.detach(), "u_grad": s["u"].grad, "p_grad": s["p"].grad}


def work(case):
    n = sum(_sizes(case))
    if case["do"] == "run":
        attempts = n * TO_THE_END[case["stage"]][1]
    else:
        attempts = n * STAGES[case["stage"]][0] * case.get("steps", 1)
    if case["do"] == "diff":
        # the forward attempt, its replay, and the adjoint of its stages (three forward's worth);
        # inputs, outputs and their adjoints
        return {"bytes": n * 8 * (27 + 4 * 15), "flops": attempts * 5 * ATTEMPT_FLOPS}
    return {"bytes": 2 * 216 * n, "flops": attempts * ATTEMPT_FLOPS}


def exact(case, seed):
    return None
