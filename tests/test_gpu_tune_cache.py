"""The cache of tuned launch shapes (sg_autotune, SG_TUNE_FILE): a shape belongs to the device, the levels, the periodic
axes and the stencil radius it was tuned with, and a line that holds chain limits in an earlier unit gives only what has
kept its meaning.  In processes of their own, since the cache lives as long as the process."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import json, os, sys
sys.path.insert(0, %r)
sys.path.insert(0, %r)
import torch
import samurai_gb300 as sg
from advection_cases import shapes_2d
NAME = torch.cuda.get_device_name(0).replace(" ", "_")
shape = lambda *a, **k: sg.MRMesh(2, *a, **k).launch_shape()  # noqa: E731
both = {"plain": ((3, 7), {}), "x": ((3, 7), dict(periodic=(True, False))), "xy": ((3, 7), dict(periodic=(True, True))),
        "wide": ((3, 7, 2), {})}
shapes = lambda: {k: shape(*a, **kw) for k, (a, kw) in both.items()}  # noqa: E731
""" % (ROOT, os.path.join(ROOT, "tests"))


def run(code, tune_file=None):
    env = {k: v for k, v in os.environ.items() if not k.startswith("SG_")}
    if tune_file:
        env["SG_TUNE_FILE"] = str(tune_file)
    r = subprocess.run([sys.executable, "-c", HEAD + code], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.strip().splitlines()[-1])


TUNE = """
defaults = shapes()
s = sg.AdvectionSim(2, 3, 7)
lv, co, _ = s.cells()
s.set_cell_values(shapes_2d(61, 4, 4)(lv, co))
s.adapt(1e-4, 2.0)
s.autotune(1e-4, 2.0, (1.0, 0.5), 0.5 / 128, steps=2)
print(json.dumps({"defaults": defaults, "chosen": s.mesh.launch_shape(), "later": shapes()}))
"""


def test_a_tuned_shape_stays_with_its_kind_of_mesh(tmp_path):
    path = tmp_path / "tunings"
    got = run(TUNE, path)
    assert got["later"]["plain"] == got["chosen"]
    for kind in ("x", "xy", "wide"):
        assert got["later"][kind] == got["defaults"][kind], kind
    # the same from the file, in another process
    again = run("print(json.dumps(shapes()))", path)
    assert again == got["later"]


def test_lines_with_limits_of_an_earlier_unit(tmp_path):
    """device dim min max block max_blocks and three limits in words per level: block, grid limit and the choice of
    graph apply to every mesh of the levels as before, the limits do not"""
    defaults = run("print(json.dumps(shapes()))")
    path = tmp_path / "tunings"
    name = run("print(json.dumps(NAME))")
    path.write_text("%s 2 3 7 128 608 1024 0 32 1 0\n" % name)
    got = run("print(json.dumps(shapes()))", path)
    for kind, was in defaults.items():
        assert got[kind] == dict(was, block=128, max_blocks=608, graphed_adapt=True, level_pairs=False), kind


def test_lines_that_are_no_shape_are_skipped(tmp_path):
    defaults = run("print(json.dumps(shapes()))")
    name = run("print(json.dumps(NAME))")
    path = tmp_path / "tunings"
    path.write_text("\n%s 2 3 7 100 608 0 0 0 0 0\nshape2 %s 2 3 7 0 1 33 608 0 0 0 0 0\nshape2 %s 2 3\n%s\n"
                    "shape2 %s 2 3 7 3 1 512 304 5000 2500 0 0 1\n" % (name, name, name, "x" * 3000, name))
    got = run("print(json.dumps(shapes()))", path)
    assert got["xy"] == dict(defaults["xy"], block=512, max_blocks=304, fuse_mesh_words=5000, fuse_field_words=2500, fuse_max_words=0)
    for kind in ("plain", "x", "wide"):
        assert got[kind] == defaults[kind], kind
