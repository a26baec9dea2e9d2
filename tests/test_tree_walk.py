"""The packed tree's walk (csrc/tree.cuh) on the CPU: its segments end for
every box, and the warps that share a query block find every pair once,
whatever boxes each of them walks with (a warp forms its boxes from the time
of impact stored when it starts, which another query lowers meanwhile)."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TREE = os.path.join(os.path.dirname(HERE), "ipc_warp_b200", "csrc", "tree.cuh")
LIMIT = 200_000  # meetings of a warp's lanes; the longest walk here has about 20,000


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    src = open(TREE).read()
    cut = re.search(r"// -+ refit\n.*?(?=// -+ traversal\n)", src, re.S)
    src = src.replace(cut.group(0), "").replace("#pragma once", "").replace('#include "common.cuh"', "")
    src = re.sub(r"inline float4\* memory\(.*?\n}\n\ninline View view\(.*?\n}\n", "", src, flags=re.S)
    src, n = re.subn(r'asm volatile\("redux\.sync\.(min|max)\.f32 %0, %1, 0xffffffff;" : "=f"\(r\) : "f"\(v\)\);',
                     lambda m: f"r = ::warp::redux(v, {'true' if m.group(1) == 'min' else 'false'});", src)
    assert n == 2
    d = tmp_path_factory.mktemp("walk")
    text = open(os.path.join(HERE, "warp_walk.cpp")).read().replace("@TREE@", src)
    (d / "walk.cpp").write_text(text)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(d / "walk.so"), str(d / "walk.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "walk.so"))
    f, i = np.ctypeslib.ndpointer(np.float32, flags="C"), np.ctypeslib.ndpointer(np.int32, flags="C")
    lib.segments.argtypes = [f, f, ctypes.c_long, i]
    lib.pairs.argtypes = [ctypes.c_int, f, f, ctypes.c_int, f, f, ctypes.c_long, i, ctypes.c_int]
    return lib


def _row(rng):
    lo = np.arange(32)[:, None] * np.float32([0.1, 0, 0]) + rng.uniform(0, 0.05, (32, 3))
    return lo.astype(np.float32), (lo + 0.1).astype(np.float32)


@pytest.mark.parametrize("size", [0.0, 1.0, 1e3, 1e18, 3e19, 1e20, 1e30, 3e38, np.inf, np.nan])
@pytest.mark.parametrize("kind", ["one", "apart", "scattered"])
def test_segments_end(walk, size, kind):
    rng = np.random.default_rng(1)
    lo, hi = _row(rng)
    if kind == "one":  # one primitive swept far
        hi[7] = size
    elif kind == "apart":  # neighbours on both sides of the origin
        lo[1::2], hi[1::2] = -size, 0.0
        lo[::2], hi[::2] = 0.0, size
    else:
        c = (rng.uniform(-0.5, 0.5, (32, 3)) * size).astype(np.float32)
        lo, hi = lo + c, hi + c
    ends = np.zeros(64, np.int32)
    n = walk.segments(lo, hi, LIMIT, ends)
    assert 1 <= n <= 32
    assert (np.diff(np.concatenate([[0], ends[:n]])) > 0).all() and ends[n - 1] == 32


@pytest.mark.parametrize("nsub", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("n, way, jump", [(33, 1, False), (1000, -1, False), (1500, 1, False), (1500, -1, True)])
def test_shared_block_finds_every_pair_once(walk, nsub, n, way, jump):
    rng = np.random.default_rng(n)
    p = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    p = p[np.argsort(p[:, 0])]
    lo, hi = p - np.float32(0.04), p + np.float32(0.04)
    # a cluster that sweeps along the curve, so a longer sweep meets more blocks
    q = rng.uniform([0.4, 0.4, 0.4], [0.6, 0.6, 0.6], (32, 3)).astype(np.float32)
    d = (rng.uniform([0.3, -0.05, -0.05], [0.35, 0.05, 0.05], (32, 3)) * [way, 1, 1]).astype(np.float32)
    if jump:  # and a few far from the rest: several segments
        q[27:] -= np.float32([0.3, 0.3, 0.3])
    # warp s sweeps to its own time
    t = np.linspace(1.0, 0.1, nsub).astype(np.float32)[rng.permutation(nsub)]
    end = q + t[:, None, None] * d
    qlo, qhi = np.minimum(q, end) - np.float32(0.01), np.maximum(q, end) + np.float32(0.01)
    out = np.zeros((400_000, 2), np.int32)
    m = walk.pairs(n, lo, hi, nsub, qlo, qhi, LIMIT, out.reshape(-1), len(out))
    assert 0 <= m <= len(out)
    found = [tuple(r) for r in out[:m]]
    assert len(set(found)) == m  # none twice

    def meets(s):
        a, b = qlo[s][:, None], qhi[s][:, None]
        return {tuple(r) for r in np.argwhere((a <= hi[None]).all(2) & (lo[None] <= b).all(2))}

    every = [meets(s) for s in range(nsub)]
    assert set.intersection(*every) <= set(found) <= set.union(*every)
