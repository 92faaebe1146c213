"""Runs a Python snippet on the product library over the fake CUDA runtime
(fake_cudart.cpp): two devices without a GPU, no kernel executed, every launch
checked against the attributes set on its device and recorded."""
import json
import os
import subprocess
import sys

import pytest

TESTS = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(TESTS)
PRELUDE = """
import json, re, sys
import numpy as np
import gpue_b200 as G
out = {}

def psi(n, dim=2):
    return np.full((n,) * dim, 0.1 + 0.0j)
"""


def build(tmp):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    so = os.path.join(str(tmp), "libfake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC",
                    "-I" + os.path.join(cuda, "include"), "-o", so,
                    os.path.join(TESTS, "fake_cudart.cpp")], check=True)
    return so


@pytest.fixture(scope="session")
def fake(tmp_path_factory):
    """run(code, **env) -> (the snippet's `out` dict, its launches)."""
    tmp = tmp_path_factory.mktemp("fake")
    so = build(tmp)

    def run(code, **env):
        log = os.path.join(str(tmp), "launches.txt")
        if os.path.exists(log):
            os.remove(log)
        e = dict(os.environ, LD_PRELOAD=so, FAKE_CUDART_LOG=log, PYTHONPATH=ROOT, **env)
        r = subprocess.run([sys.executable, "-c", PRELUDE + code + "\nprint(json.dumps(out))"],
                           env=e, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        launches = []
        if os.path.exists(log):
            for line in open(log):
                d, name, grid, threads, smem, cluster, coop, status = line.split()
                launches.append({"device": int(d), "kernel": name, "grid": int(grid),
                                 "threads": int(threads), "smem": int(smem),
                                 "cluster": int(cluster), "coop": int(coop),
                                 "status": int(status)})
        return json.loads(r.stdout.strip().splitlines()[-1]), launches

    return run
