"""Which faces share a launch (csrc/device/face_groups.hpp), against the points
the kernels reach: random faces on all sides of a few blocks, inner faces in
every orientation and with both signs along each axis, enumerated point by point
as k_bc and k_inner map them."""
import itertools
import random
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    from openstc_b200.build import _cuda_home

    exe = tmp_path_factory.mktemp("faces") / "faces"
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", str(ROOT / "openstc_b200" / "csrc"), "-I",
                    str(_cuda_home() / "include"), str(ROOT / "tests" / "face_groups.cpp"), "-o", str(exe)], check=True)

    def run(faces):
        text = "\n".join(f["kind"] + " " + " ".join(str(v) for v in flat(f)) for f in faces)
        out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
        assert len(out) == len(faces)
        return [int(v) for v in out]

    return run


def flat(f):
    keys = ["g", "block", "face", "start", "end"] if f["kind"] == "b" else [
        "g", "block", "target", "face", "start", "loop_dir", "tstart", "tloop_dir", "src_tar", "n_point"]
    for k in keys:
        yield from f[k] if isinstance(f[k], list) else [f[k]]


def points(f):
    """The (block, point)s that the face's kernel reads or writes."""
    out = set()
    if f["kind"] == "b":
        ranges = [range(f["start"][q], f["end"][q] + 1) for q in range(3)]
        for p in itertools.product(*ranges):
            for layer in range(-f["g"], f["g"] + 1):
                x = list(p)
                x[f["face"]] += layer
                out.add((f["block"], *x))
        return out
    spans = []
    for q in range(3):
        wide = f["g"] if q != f["face"] and f["n_point"][q] > 1 else 0
        spans.append(range(-wide, f["n_point"][q] + wide))
    if 0 in f["n_point"]:
        return out
    for nn in itertools.product(*spans):
        d = [f["loop_dir"][q] * nn[q] for q in range(3)]
        out.add((f["block"], *[f["start"][q] + d[q] for q in range(3)]))
        out.add((f["target"], *[f["tstart"][q] + f["tloop_dir"][q] * d[f["src_tar"][q]] for q in range(3)]))
    return out


def random_faces(rng, kind, n, g):
    faces = []
    for _ in range(n):
        face = rng.randrange(3)
        f = dict(kind=kind, g=g, block=rng.randrange(3), face=face)
        lo, size = [rng.randint(-2, 9) for _ in range(3)], [rng.randint(0 if rng.random() < 0.1 else 1, 5) for _ in range(3)]
        if kind == "b":
            size[face] = min(size[face], 1)
            f.update(start=lo, end=[a + s - 1 for a, s in zip(lo, size)])
        else:
            src_tar = rng.sample(range(3), 3)
            f.update(target=rng.randrange(3), start=lo, loop_dir=[rng.choice([-1, 1]) for _ in range(3)],
                     tstart=[rng.randint(-2, 9) for _ in range(3)], tloop_dir=[rng.choice([-1, 1]) for _ in range(3)],
                     src_tar=src_tar, n_point=size)
        faces.append(f)
    return faces


@pytest.mark.parametrize("kind,g", [("b", 2), ("b", 3), ("i", 0), ("i", 2)])
def test_faces_of_a_launch_touch_no_common_point_and_keep_their_order(launches, kind, g):
    rng = random.Random(17 + g)
    shared = 0
    for _ in range(40):
        faces = random_faces(rng, kind, rng.randint(1, 10), g)
        launch, touched = launches(faces), [points(f) for f in faces]
        for q, e in itertools.combinations(range(len(faces)), 2):
            if launch[q] < 0 or launch[e] < 0:
                assert not (touched[q] if launch[q] < 0 else touched[e])
            elif touched[q] & touched[e]:
                assert launch[q] < launch[e], (faces[q], faces[e])
            else:
                shared += launch[q] == launch[e]
    assert shared > 40  # the grouping does group
