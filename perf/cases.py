"""Performance cases of the renderer: what a user has it do, through the
package's public calls.

A case is a plain dict.  "call" names the entry point: "trace"
(Renderer.trace into device buffers), "render" (Renderer.render_host: trace,
colour, image on the host), "batch" (Batch.launch over many frames) and
"grad" (Renderer.l2_grad).  The other entries are kt_frame_desc fields; the
seed turns the camera and shifts its inclination and the spin a little, as
the frames of an animation or a parameter scan do.

There is no exact(): a trace's numbers are those of the adaptive integrator's
own accept/reject sequence, which every rounding moves (two builds of the
same renderer differ by 1e-6 in a pixel's redshift at the median, and by
whole disk radii at the critical curve), so 64-bit arithmetic in another
order is no closer to a true value than the renderer is; the FP64 records are
defined bit for bit instead.
"""
import random

import torch

import kerrtracecpp2_b200 as kt

BL, KS = 1, 0
RK4, DOPRI5 = 0, 1
FP64, MIXED, SMOOTH = 0, 1, 2

# The metric and camera of a frame: (a, Q, Lambda, theta, r_obs, fov, disk_out).
KERR_HALF = dict(a=0.5, Q=0.0, Lambda=0.0, theta_deg=80.0, r_obs=40.0, fov_deg=45.0, disk_out=12.0)
KERR_FAST = dict(a=0.998, Q=0.0, Lambda=0.0, theta_deg=80.0, r_obs=40.0, fov_deg=30.0, disk_out=12.0)
KNDS = dict(a=0.9, Q=0.3, Lambda=1e-4, theta_deg=85.0, r_obs=60.0, fov_deg=30.0, disk_out=20.0)
KN = dict(a=0.7, Q=0.1, Lambda=0.0, theta_deg=70.0, r_obs=50.0, fov_deg=30.0, disk_out=15.0)


def _case(call, width, height, metric, chart, integrator=RK4, tol=1e-7, precision=FP64, bundles=0,
          spp=1, frames=1, max_steps=500000):
    return dict(call=call, width=width, height=height, chart=chart, integrator=integrator, tol=tol,
                precision=precision, bundles=bundles, spp=spp, frames=frames, max_steps=max_steps, **metric)


def listed():
    return [
        # a thumbnail, as a user interface asks for while a slider moves
        dict(_case("trace", 48, 27, KERR_HALF, KS), name="trace_ks_48x27"),
        # the preview size: Kerr, KS chart, the command line's default integrator
        dict(_case("trace", 320, 180, KERR_HALF, KS), name="trace_ks_320x180"),
        # the command line's default frame at 720p: trace, colour with a
        # background, image on the host
        dict(_case("render", 1280, 720, KERR_FAST, KS), name="render_ks_1280x720"),
        # the headline frame: Kerr-Newman-de Sitter, BL chart, DOPRI5 at 1e-10
        dict(_case("trace", 1280, 720, KNDS, BL, DOPRI5, 1e-10), name="trace_bl_dopri5_1280x720"),
        # Kerr in the BL chart (--bl), an odd size
        dict(_case("trace", 641, 359, KERR_FAST, BL), name="trace_bl_rk4_641x359"),
        # Jacobi bundles (--bundles): magnification per pixel
        dict(_case("trace", 960, 540, dict(KERR_FAST, theta_deg=60.0), BL, bundles=1),
             name="trace_bundle_960x540"),
        # mixed precision at the headline tolerance (analytic gradient in FP64)
        dict(_case("trace", 1280, 720, KNDS, BL, DOPRI5, 1e-10, MIXED), name="trace_mixed_dopri5_1280x720"),
        # mixed precision at the default tolerance (FP32 far field), KS chart
        dict(_case("trace", 512, 512, KN, KS, precision=MIXED), name="trace_mixed_ks_512x512"),
        # a scan over spin, inclination and Lambda as one batch (both charts)
        dict(_case("batch", 256, 256, KN, KS, frames=12), name="batch_12x256x256"),
        # gradient of an image loss, the KS chart's default integrator
        dict(_case("grad", 512, 512, KN, KS), name="grad_ks_512x512"),
        # gradient with DOPRI5 in the BL chart
        dict(_case("grad", 640, 360, KNDS, BL, DOPRI5, 1e-10), name="grad_bl_dopri5_640x360"),
        # gradient of a bundle frame, the magnification in the loss
        dict(_case("grad", 320, 180, dict(KERR_FAST, theta_deg=60.0), BL, bundles=1),
             name="grad_bundle_320x180"),
    ]


# Pixels of the smallest and largest case of each kind of work.
_SPAN = {"trace_ks": (1296, 921600), "trace_bl": (1296, 921600), "trace_bundle": (1296, 129600),
         "trace_mixed": (1296, 921600), "render": (1296, 921600), "batch": (4096, 65536),
         "grad": (1296, 262144), "grad_bundle": (1296, 57600)}


def draw(rng):
    kind = rng.choice(sorted(_SPAN))
    lo, hi = _SPAN[kind]
    n = lo * (hi / lo) ** rng.random()
    aspect = rng.choice([1.0, 4.0 / 3.0, 16.0 / 9.0])
    w = max(16, int(round((n * aspect) ** 0.5)))
    h = max(9, min(int(n / w), hi // w))
    metric = dict(a=round(rng.uniform(0.0, 0.998), 4), Q=rng.choice([0.0, round(rng.uniform(0.0, 0.05), 4)]),
                  Lambda=0.0, theta_deg=round(rng.uniform(20.0, 88.0), 2),
                  r_obs=round(rng.uniform(20.0, 100.0), 2), fov_deg=rng.choice([20.0, 30.0, 45.0]),
                  disk_out=rng.choice([12.0, 15.0, 20.0]))
    dp = rng.random() < 0.5
    tol = rng.choice([1e-8, 1e-9, 1e-10]) if dp else rng.choice([1e-6, 1e-7, 1e-8])
    lam = rng.choice([0.0, 1e-5, 1e-4])
    intg = DOPRI5 if dp else RK4
    if kind in ("trace_ks", "render"):
        tol = rng.choice([1e-6, 1e-7, 1e-8])
        return _case("trace" if kind == "trace_ks" else "render", w, h, metric, KS, RK4, tol,
                     spp=rng.choice([1, 1, 2]) if kind == "render" and n < hi / 4 else 1)
    if kind == "trace_bl":
        return _case("trace", w, h, dict(metric, Lambda=lam), BL, intg, tol)
    if kind in ("trace_bundle", "grad_bundle"):
        # fast spin, and a step cap as a program sets it: a bundle ray that
        # runs out near the equator meets no escape test and ends at the cap
        metric.update(a=round(rng.uniform(0.9, 0.998), 4), theta_deg=round(rng.uniform(40.0, 62.0), 2))
        return _case("trace" if kind == "trace_bundle" else "grad", w, h, metric, BL, RK4, 1e-7, bundles=1,
                     max_steps=1000)
    if kind == "trace_mixed":
        chart = rng.choice([KS, BL])
        return _case("trace", w, h, dict(metric, Lambda=lam if chart == BL else 0.0), chart,
                     intg if chart == BL else RK4, tol, MIXED)
    if kind == "batch":
        return _case("batch", w, h, metric, KS, RK4, 1e-7, frames=rng.randint(2, 12))
    chart = rng.choice([KS, BL])
    return _case("grad", w, h, dict(metric, Lambda=lam if chart == BL else 0.0), chart,
                 intg if chart == BL else RK4, tol)


_FIELDS = ("a", "Q", "Lambda", "theta_deg", "r_obs", "fov_deg", "disk_out", "width", "height", "chart",
           "integrator", "tol", "precision", "bundles", "max_steps")

_one = {}


def _renderer():
    """The renderer that the program keeps (one per device)."""
    if "r" not in _one:
        _one["r"] = kt.Renderer(torch.cuda.current_device())
    return _one["r"]


def _background():
    if "bg" not in _one:
        _one["bg"] = kt.starfield(0)
    return _one["bg"]


def _desc(case, rng, **kw):
    f = {k: case[k] for k in _FIELDS}
    f["a"] = min(0.998, max(0.0, f["a"] + rng.uniform(-0.004, 0.004)))
    f["theta_deg"] += rng.uniform(-0.5, 0.5)
    f["phi_deg"] = rng.uniform(0.0, 360.0)
    f.update(kw)
    return kt.frame_desc(**f)


def _scan(case, rng):
    """The frames of a batch: spin and inclination over their ranges, every
    other frame with Lambda = 1e-4 (which takes the BL chart)."""
    n = case["frames"]
    out = []
    for i in range(n):
        t = (i + 0.5) / n
        out.append(_desc(case, rng, a=0.95 * t + rng.uniform(-0.02, 0.02), theta_deg=85.0 - 60.0 * t,
                         r_obs=case["r_obs"] * (0.8 + 0.4 * t), Lambda=1e-4 if i % 2 else 0.0))
    return out


def prepare(case, seed):
    rng = random.Random(seed)
    r = _renderer()
    if case["call"] == "batch":
        descs = _scan(case, rng)
        n = case["width"] * case["height"]
        whole = r.alloc(n * len(descs))  # every frame's records, one buffer a field
        outs = [{k: v[i * n:(i + 1) * n] for k, v in whole.items()} for i in range(len(descs))]
        return {"call": "batch", "batch": r.batch(descs, outs), "out": whole}
    desc = _desc(case, rng)
    n = case["width"] * case["height"]
    if case["call"] == "trace":
        return {"call": "trace", "r": r, "desc": desc, "out": r.alloc(n)}
    if case["call"] == "render":
        return {"call": "render", "r": r, "desc": desc, "bg": _background(), "spp": case["spp"],
                "cp": kt.color_params()}
    # the target image of the loss: the smooth tracer at another spin and inclination
    f = {k: getattr(desc, k) for k in _FIELDS}
    f.update(phi_deg=desc.phi_deg, precision=SMOOTH, a=max(0.0, min(0.998, desc.a - 0.01)),
             theta_deg=desc.theta_deg + 1.0)
    target = r.trace(kt.frame_desc(**f))
    return {"call": "grad", "r": r, "desc": desc, "target": target, "out": r.alloc(n),
            "w_m": 0.01 if case["bundles"] else 0.0}


def run(state):
    if state["call"] == "batch":
        state["batch"].launch()
        return state["out"]
    if state["call"] == "trace":
        return state["r"].trace(state["desc"], state["out"])
    if state["call"] == "render":
        return state["r"].render_host(state["desc"], state["cp"], state["bg"], state["spp"])
    loss, grad, stats = state["r"].l2_grad(state["desc"], state["target"], 1.0, 0.01, state["out"],
                                           w_m=state["w_m"])
    return {"loss": loss, "grad": grad, "grad_pixels": stats["grad_pixels"], "out": state["out"]}


# Arithmetic of one adaptive attempt (+, -, *, / and sqrt 1 flop, fma 2,
# sincos 70): BL right-hand side 447 (211 of arithmetic, 26 divisions, three
# sincos), KS 820 (seven metric evaluations), a bundle's 2000, the analytic
# gradient 250; DOPRI5 takes 6 of them, RK4 step doubling 10 and one more per
# accepted step.
_RHS = {"bl": 447.0, "ks": 820.0, "bundle": 2000.0, "analytic": 250.0}


def work(case):
    n = float(case["width"] * case["height"] * case["frames"] * case["spp"])
    dp = case["integrator"] == DOPRI5 and case["chart"] == BL
    # adaptive attempts per ray at the reference tolerances (measured means)
    attempts = 145.0 * (1e-10 / case["tol"]) ** 0.2 if dp else 62.0 * (1e-7 / case["tol"]) ** 0.2
    if case["bundles"]:
        attempts = 75.0 * (1e-7 / case["tol"]) ** 0.2
    kind = "ks" if case["chart"] == KS else "bl"
    if case["bundles"]:
        kind = "bundle"
    if case["precision"] == MIXED or case["call"] == "grad":
        kind = "analytic"
    flops = n * attempts * ((6.0 if dp else 11.0) * _RHS[kind] + 330.0)
    out = 58.0 * n  # the records: six float64, two 32-bit counters, two bytes
    if case["call"] == "render":
        return {"bytes": 3.0 * case["width"] * case["height"] + 3.0 * 2048 * 1024, "flops": flops}
    if case["call"] == "grad":
        # forward and the reverse sweep over it (about twice its arithmetic);
        # the target's class, redshift, radius and magnification are read
        return {"bytes": out + 25.0 * n, "flops": 3.0 * flops}
    return {"bytes": out, "flops": flops}
