"""Render iterations as a user of the framework runs them: what is timed and
how far two correct builds may differ.

A case is a command line of the renderer on a generated or predefined scene
(workload, size, techniques, path length, radii, iteration index), or a
batch of small jobs.  `prepare` writes the scene, loads it and creates the
renderer, all of which a program does once; a pass is one render iteration
and the copy of its image into page-locked host memory, which a program
does for every iteration it renders.  A pass renders the same iteration
index each time, so it gives the same image whenever it runs: the random
numbers and the radii depend on the index alone.

The seed changes the scene (materials, shapes, media, or for the meshes of
half a million triangles and more, which take seconds to write, the place of
the camera) and the random stream (-ioff).

The learned proposal (-guide) has no case: its network is trained with
float atomics, so two runs of the same build already sample other paths and
their images differ by Monte Carlo noise, not by rounding.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

from gpuupbp_b200 import batch, scenes, upbp

SIX = "upbp_bpt+surf+pp3d+pb2d+bb1d+bp2d"   # every estimator and BPT (bench.py)
ALL = "upbp_all"                            # the command line's own set: no BP2D
R2 = -0.02                                  # the box workloads' radius, of the scene radius

# Scenes: `pixels` bounds a drawn case's resolution so that it costs no more
# than the largest listed case (beam pairs grow with pixels x light paths),
# then the range of path lengths, the radius the workload is rendered with
# (0: the command line's), whether the mesh is large; and what a pass cannot
# do without: triangles, stored light vertices and beams of a light path, and
# accepted BB1D pairs over camera x light paths at the first iteration's
# radius (counts of one iteration each).  The path lengths leave room for every
# beam: past its capacity (length - 2 beams a light path) a renderer drops
# the beams that come last, in no fixed order, as the reference does.
SCENES = {
    "box_medium": dict(pixels=256 * 256, length=(4, 16), radius=R2, mesh=False, tris=1294, verts=2.8, beams=0.8,
                       pairs=3.0e-2),
    "batch_job": dict(pixels=256 * 256, length=(4, 16), radius=R2, mesh=False, tris=30000, verts=2.9, beams=1.2,
                      pairs=2.5e-2),
    "glass_box": dict(pixels=256 * 256, length=(4, 12), radius=R2, mesh=False, tris=2600, verts=2.9, beams=0.8,
                      pairs=3.0e-2),
    "fog_box": dict(pixels=160 * 160, length=(7, 12), radius=R2, mesh=False, tris=1294, verts=3.0, beams=3.0,
                    pairs=3.0e-2),
    "media_field": dict(pixels=1280 * 720, length=(6, 12), radius=0.0, mesh=True, tris=1638484, verts=0.54,
                        beams=0.3, pairs=1.7e-4),
    "media_field_env": dict(pixels=960 * 540, length=(6, 12), radius=0.0, mesh=True, tris=1638484, verts=0.53,
                            beams=0.29, pairs=1.7e-4),
    "dense_beams": dict(pixels=400 * 225, length=(8, 16), radius=0.0, mesh=True, tris=504514, verts=5.0, beams=3.4,
                        pairs=2.2e-2),
}
PREDEF = dict(pixels=512 * 512, length=(8, 14), radius=0.0, mesh=False, tris=32, verts=1.4, beams=0.5, pairs=1.0e-3)


def _scene(case):
    return SCENES.get(case["scene"], PREDEF)


def _case(name, scene, res, tech=ALL, length=8, iteration=0, radius=0.0, extra="", tiny=False):
    return {"name": name, "scene": scene, "width": res[0], "height": res[1], "tech": tech, "length": length,
            "iteration": iteration, "radius": radius, "extra": extra, "tiny": tiny, "jobs": 0}


def listed():
    return [
        # a preview: the smallest job of the batched workload (64 x 64), where
        # launches, host synchronisations and short kernels are the time
        _case("preview 64x64", "box_medium", (64, 64), radius=R2),
        # the plain small workload: unit box around one fog sphere, 256 x 256
        _case("box 256x256", "box_medium", (256, 256), radius=R2),
        # the large jobs of the batched workload, at an odd size, long paths
        _case("job 367x293", "batch_job", (367, 293), length=14, radius=R2, iteration=3),
        # the benchmark: 1.64M triangles, 20 media, every estimator
        _case("media field 1280x720", "media_field", (1280, 720), tech=SIX, length=12),
        # the same scene as a smaller, ragged frame, later in a render (smaller radii)
        _case("media field 641x359", "media_field", (641, 359), tech=SIX, length=10, iteration=40),
        # path tracing alone: no photon maps, the ray casts and connections are all
        _case("bpt 960x540", "media_field", (960, 540), tech="upbp_bpt", length=12),
        # the thick forward-scattering medium: many short beams, long paths
        _case("dense beams 480x270", "dense_beams", (480, 270), tech=SIX, length=16,
              extra="-r_initial_bb1d -0.004 -r_initial_bp2d -0.004"),
        # photons only (surfaces, points, point-beams), short query beams
        _case("photons 400x300", "fog_box", (400, 300), tech="upbp+surf+pp3d+pb2d", length=8, radius=R2,
              extra="-qbt S"),
        # analytic spheres: a predefined scene (a small scattering box), default settings
        _case("spheres 512x512", "predef:35", (512, 512), tech=SIX, length=12),
        # surfaces under an environment map, beams towards points, -pcpi and -pbc
        _case("sky 480x270", "media_field_env", (480, 270), tech="upbp_bpt+surf+bp2d", length=8,
              extra="-pcpi 200000 -r_initial_bp2d -0.002"),
        # many small jobs rendered together (upbp_run_batch)
        dict(_case("batch of 12", "batch_job", (160, 160), length=12, radius=R2), jobs=12),
    ]


def draw(rng):
    scene = rng.choice(sorted(SCENES) + ["box_medium", "media_field", "predef"])
    s = SCENES.get(scene, PREDEF)
    if scene == "predef":
        scene = "predef:%d" % rng.choice([0, 1, 5, 6, 7, 13, 21, 22, 28, 30, 39])
    pixels = math.exp(rng.uniform(math.log(40 * 40), math.log(s["pixels"])))
    aspect = rng.choice([1.0, 4 / 3, 16 / 9, 0.75])
    w = max(24, int(math.sqrt(pixels * aspect)))
    h = max(24, int(pixels / w))
    tech = rng.choice([ALL, SIX, SIX, "upbp_bpt", "upbp_bb1d", "upbp_surf", "upbp+pp3d+pb2d", "upbp+bp2d+pb2d"])
    extra = []
    if rng.random() < 0.25:
        extra += ["-qbt", "S"]
    if rng.random() < 0.15:
        extra += ["-pbt", "S"]
    if rng.random() < 0.25:
        extra += ["-pcpi", str(rng.randrange(max(500, w * h // 8), w * h + 1))]
    if rng.random() < 0.15:
        extra += ["-pbc", str(rng.randrange(200, max(201, w * h // 4)))]
    if rng.random() < 0.1:
        extra += ["-sn"]
    if scene == "dense_beams":
        extra += ["-r_initial_bb1d", "-0.004", "-r_initial_bp2d", "-0.004"]
    return _case("", scene, (w, h), tech=tech, length=rng.randint(*s["length"]),
                 iteration=int(math.exp(rng.uniform(0.0, math.log(200.0)))) - 1, radius=s["radius"],
                 extra=" ".join(extra)) | {"name": None}


# --------------------------------------------------------------------------- inputs

_DIR = os.path.join(tempfile.gettempdir(), "upbp_perf_scenes")


def _orbit(path, seed):
    """The scene at `path` seen from a camera of the seed's own: the .aux file
    names the camera, the mesh is shared by a hard link."""
    rng = random.Random(seed)
    out = path[:-4] + "_view%d.obj" % seed
    with open(path + ".aux") as f:
        lines = f.read().splitlines()
    rows = {ln.split()[0]: np.array([float(x) for x in ln.split()[1:4]]) for ln in lines if ln.startswith("TM_ROW")}
    a = rng.uniform(-0.25, 0.25)
    turn = np.array([[math.cos(a), 0.0, math.sin(a)], [0.0, 1.0, 0.0], [-math.sin(a), 0.0, math.cos(a)]])
    scale = rng.uniform(0.9, 1.0)
    if not os.path.exists(out):
        try:
            os.link(path, out)
        except FileExistsError:
            pass
    with open(out + ".aux", "w") as f:
        for ln in lines:
            key = ln.split()[0] if ln.split() else ""
            if key in rows:
                v = turn @ rows[key] * (scale if key == "TM_ROW3" else 1.0)
                ln = "%s %.7f %.7f %.7f" % (key, *v)
            f.write(ln + "\n")
    return out


def _args(case, seed):
    scene = case["scene"]
    if scene.startswith("predef:"):
        where = ["-s", scene.split(":")[1]]
    elif _scene(case)["mesh"]:
        where = ["-s", "-1", _orbit(scenes.write_workload(scene, _DIR, tiny=case["tiny"]), seed)]
    else:
        where = ["-s", "-1", scenes.write_workload(scene, _DIR, seed=seed, tiny=case["tiny"])]
    args = where + case["extra"].split() + ["-a", case["tech"], "-l", str(case["length"]), "-r", "%dx%d" % (case["width"], case["height"]),
                    "-ioff", str(1000 * (seed % 100000))]
    if case["radius"]:
        args += ["-r_initial", str(case["radius"]), "-r_alpha", "0.75"]
    return args


def _host_image(r):
    return torch.zeros((r.height, r.width, 3), dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    if case["jobs"]:
        jobs = []
        for k in range(case["jobs"]):  # uneven sizes and path lengths, as the batched workload draws them
            rng = random.Random(k)
            side = rng.choice([64, 96, 128, case["width"]])
            jobs.append(_args(dict(case, width=side, height=side, length=rng.randint(4, case["length"])),
                              seed * 64 + k))
        b = batch.Batch(jobs)
        return {"batch": b, "iteration": case["iteration"], "images": [_host_image(r) for r in b.renderers]}
    r = upbp.Renderer(_args(case, seed))
    return {"renderer": r, "iteration": case["iteration"], "image": _host_image(r)}


def run(state):
    if "batch" in state:
        b = state["batch"]
        b.run_iteration(state["iteration"], workers=4)
        return [r.iteration_image(out=img) for r, img in zip(b.renderers, state["images"])]
    r = state["renderer"]
    r.run_iteration(state["iteration"])
    return r.iteration_image(out=state["image"])


# --------------------------------------------------------------------------- what it costs, how far it may be off

def work(case):
    """Bytes: the scene read once (92 B a triangle: corners, normals, ids),
    the light vertices (80 B) and beams (128 B) written and read once, the
    image written.  Operations: about 500 for each bounce of a path (three a
    path) and 200 for each accepted pair of a query beam and a photon beam."""
    s, n = _scene(case), max(1, case["jobs"])
    px = case["width"] * case["height"]
    beams = any(t in case["tech"] for t in ("bb1d", "bp2d", "all"))
    records = 2 * 80 * s["verts"] + (2 * 128 * s["beams"] if beams else 0)
    pairs = s["pairs"] * float(px) ** 2 if "bb1d" in case["tech"] or "all" in case["tech"] else 0.0
    if case["jobs"]:
        px *= 0.5  # the jobs are 64^2 .. width x height
        pairs *= 0.35
    return {"bytes": n * (92.0 * s["tris"] + px * (records + 12.0)), "flops": n * (500.0 * 2 * px * 3 + 200.0 * pairs)}


def tolerance(case):
    """Sums in another order and evaluations with other roundings, the paths
    being the same.  Rendering twice (the float atomics land in another order)
    differs by up to 1.2e-6 (max 1e-5); a build without fused multiply-adds
    differs by up to 6.5e-6 (max 1.3e-3) on cases where it traces the same
    paths.  Where its roundings send one path another way, single pixels
    change by more than their value: the random decisions of a path are part
    of what a seed stands for, so that is not allowed for here."""
    return {"rel": 3e-5, "max": 5e-3}


def exact(case, seed):
    """None: in 64 bits every random decision near a rounding error goes the
    other way on some paths, so such a render shows other noise, and one of
    these sizes in plain numpy takes hours."""
    return None
