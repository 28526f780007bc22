"""The order of work of an attention kernel's issuing warp (trinix_b200/csrc/attention_issue.cuh), run
on the host against a model of the barriers and copies around it."""
from __future__ import annotations

import ctypes
import os
import random
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "trinix_b200", "csrc")
WRONG = ["", "a barrier was lapped", "a stage was overwritten", "a stage was released twice",
         "wrong order", "deadlock", "unfinished"]


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("model") / "issue.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-Wno-unknown-pragmas",
                           "-I", CSRC, "-o", lib, os.path.join(HERE, "attention_issue_model.cpp")])
    return ctypes.CDLL(lib).issue_model


def _item(rng, kind):
    """(visits, first, end of this Q tile's): as the items of a launch have them."""
    n = rng.choice([1, 2, 3, 4, 5, 9])
    if kind == "mixed":
        kind = rng.choice(["whole", "no keys", "empty", "late", "early"])
    return {"whole": (n, 0, n), "no keys": (0, 0, 0), "empty": (n, 0, 0),
            "late": (n, 1, n) if n > 1 else (n, 0, n),
            "early": (n, 0, n - 1) if n > 1 else (n, 0, n)}[kind]


@pytest.mark.parametrize("kinds", [["whole"], ["early"], ["late"], ["empty"], ["empty", "late"],
                                   ["mixed"]], ids="-".join)
def test_issue_order(model, kinds):
    """Lists of up to five items, 3000 of each kind, copies landing in random order."""
    rng = random.Random(len(kinds[0]))
    for seed in range(3000):
        items = [_item(rng, rng.choice(kinds)) for _ in range(rng.randint(1, 5))]
        cols = [(ctypes.c_int * len(items))(*c) for c in zip(*items)]
        wrong = model(len(items), *cols, ctypes.c_uint64(seed))
        assert wrong == 0, (WRONG[wrong], items, seed)
