"""Writes tests/golden/hit_order.npz: rays and their hits for tests/test_gpu_hit_order.py.

Needs a GPU and two built trees: A, whose hits are recorded (commit 76642e9, the last one with the slots of
all nodes as the tree builder lists them and one offset for all box tests), and B, another build.  Taken
are the first 500 rays of a large set that the two answer differently, of each kind of query, and 300 others.
Run from the repository root: python tests/golden/make_hit_order.py A B
"""
import importlib
import os
import subprocess
import sys
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
SETS = {"crowd": (1 << 20, 23, 5.0), "coincident": (24 << 20, 29, 1.0)}  # rays, seed, extent


def trace(path):
    """All rays of both scenes with the package of the tree in the working folder."""
    sys.path[:0] = [os.getcwd(), os.path.dirname(HERE)]
    T = importlib.import_module("test_gpu_hit_order")
    out = {}
    for name, (n, seed, extent) in SETS.items():
        scene, r = getattr(T, name)(), T.rays(n, seed, extent)
        for kind in ("any", "closest"):
            hits, inst = scene.trace_host(r, any_hit=kind == "any", incoherent=True)
            out[f"{name}_{kind}"] = np.column_stack([hits.view(np.uint32), inst])
    np.savez(path, **out)


def main(a, b):
    got = []
    with tempfile.TemporaryDirectory() as tmp:
        for k, tree in enumerate((a, b)):
            path = os.path.join(tmp, f"{k}.npz")
            subprocess.run([sys.executable, os.path.abspath(__file__), "--trace", path], cwd=tree, check=True)
            got.append(dict(np.load(path)))
    sys.path[:0] = [os.path.abspath(a), os.path.dirname(HERE)]
    T = importlib.import_module("test_gpu_hit_order")
    out = {}
    for name, (n, seed, extent) in SETS.items():
        same, pick = np.ones(n, bool), []
        for kind in ("any", "closest"):
            d = (got[0][f"{name}_{kind}"] != got[1][f"{name}_{kind}"]).any(1)
            print(name, kind, int(d.sum()), "of", n, "differ")
            same &= ~d
            pick.append(np.flatnonzero(d)[:500])
        pick = np.concatenate(pick + [np.flatnonzero(same)[:300]])
        out[name + "_rays"] = T.rays(n, seed, extent)[pick]
        for kind in ("any", "closest"):
            out[f"{name}_{kind}"] = got[0][f"{name}_{kind}"][pick]
    np.savez_compressed(os.path.join(HERE, "hit_order.npz"), **out)


if __name__ == "__main__":
    trace(sys.argv[2]) if sys.argv[1] == "--trace" else main(*sys.argv[1:3])
