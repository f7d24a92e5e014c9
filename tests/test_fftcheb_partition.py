"""The transport's split of its workspace (csrc/fftcheb_partition.cuh), compiled
for the host: the stores and the transform buffers stay within the bound, and a
bound that was enough stays enough."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
GB = 1 << 30


@pytest.fixture(scope="module")
def partition(tmp_path_factory):
    exe = tmp_path_factory.mktemp("partition") / "probe"
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O1", "-Wall", "-Werror",
                    str(ROOT / "tests" / "cpp" / "partition_probe.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)

    def ask(cases):
        keys = ("workspace", "fixed", "brows", "b", "R", "M", "cplx", "bastin", "part", "sections")
        text = "\n".join(" ".join(str(int(c[k])) for k in keys) for c in cases)
        out = subprocess.run([str(exe)], input=text, check=True, capture_output=True, text=True)
        rows = [list(map(int, line.split())) for line in out.stdout.splitlines()]
        assert len(rows) == len(cases)
        names = ("fit", "sec_brows", "sections", "chunk_rows", "e_bytes", "ctas")
        return [dict(zip(names, r)) for r in rows]

    return ask


def _store(c):
    return 2 * c["M"] * c["b"] * 3 * c["R"] * c["cplx"]


def _per_row(c):
    """A row in the cuFFT stage: both sides' points and as much again for cuFFT."""
    return 2 * 2 * (4 if c["bastin"] else 1) * c["M"] * 3 * c["R"] * 16


def _held(c, p):
    row_stage = p["e_bytes"] + p["ctas"] * c["part"] if c["part"] else 2 * p["e_bytes"]
    return c["fixed"] + p["sec_brows"] * _store(c) + row_stage


def test_a_row_of_more_than_the_cap_stays_within_the_bound(partition):
    """Bastin, 256 samples, 12,000 moments: one row's transforms are 2.2 GB, more
    than the stage's usual share, and the workspace's quarter holds them."""
    c = dict(workspace=12 * GB, fixed=GB // 4, brows=1000, b=1, R=256, M=12000, cplx=16,
             bastin=1, part=0, sections=0)
    assert 2 * GB < _per_row(c) < (c["workspace"] - c["fixed"]) // 4
    p, = partition([c])
    assert p["fit"] == 0 and p["chunk_rows"] == 1
    assert _held(c, p) <= c["workspace"]


def _enough(c):
    """What a quarter for the transforms leaves holds a block row's stores."""
    if c["workspace"] <= c["fixed"] + _store(c):
        return False
    avail = c["workspace"] - c["fixed"]
    return avail - avail // 4 >= _store(c)


def test_bounds_over_random_shapes(partition):
    rng = np.random.default_rng(1)
    cases = []
    for _ in range(4000):
        M = int(np.exp(rng.uniform(0, np.log(20000))))
        fused = int(rng.random() < 0.3)
        if fused:
            M = int(rng.choice([256, 512, 1024, 2048]))
        c = dict(b=int(rng.choice([1, 4, 5, 8, 13])), R=int(np.exp(rng.uniform(0, np.log(256)))),
                 M=M, cplx=int(rng.choice([8, 16])), part=fused * 8 * 256 * 16,
                 bastin=0 if fused else int(rng.random() < 0.5),
                 brows=int(np.exp(rng.uniform(0, np.log(200000)))),
                 sections=int(rng.choice([0, 0, 1, 3])))
        c["fixed"] = c["brows"] * c["b"] * c["R"] * c["cplx"] * 18
        c["workspace"] = c["fixed"] + int(_store(c) * np.exp(rng.uniform(np.log(0.9), np.log(1e5))))
        cases.append(c)
    fits = 0
    for c, p in zip(cases, partition(cases)):
        if _enough(c):
            assert p["fit"] == 0, c
        if p["fit"]:
            continue
        fits += 1
        assert 1 <= p["sec_brows"] <= c["brows"] and p["chunk_rows"] >= 1
        assert p["sections"] * p["sec_brows"] >= c["brows"] > (p["sections"] - 1) * p["sec_brows"]
        if c["part"]:
            # beyond the bound by a pair of sequences and one CTA's sums at most,
            # where one block row's stores take all but less than these
            spare = c["workspace"] - c["fixed"] - _store(c)
            least = 2 * c["M"] * c["cplx"] + c["part"]
            assert p["ctas"] >= 1 and p["e_bytes"] >= 2 * c["M"] * c["cplx"]
            assert _held(c, p) <= c["workspace"] + (least if spare < 2 * least else 0), (c, p)
        elif _per_row(c) <= (c["workspace"] - c["fixed"]) // 4:
            assert _held(c, p) <= c["workspace"], (c, p)
    assert fits > 2000
