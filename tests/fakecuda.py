"""Runs a piece of Python on the library in a process of its own whose CUDA runtime is
tests/fake_cuda.cpp (no device needed)."""
import functools
import json
import os
import subprocess
import sys
import tempfile
import textwrap
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = """
import ctypes, json, sys
sys.path.insert(0, {root!r})
import numpy as np
from mpsxx_gb300 import core
from mpsxx_gb300._lib import MpsxxError
from tests.fakecuda import operands
fake = ctypes.CDLL({fake!r})
fake.fake_limit.argtypes = [ctypes.c_size_t]
fake.fake_used.restype = ctypes.c_size_t

def launches(name=""):
    n = fake.fake_log(None, 0) + 1
    b = ctypes.create_string_buffer(n)
    fake.fake_log(b, n)
    return [x for x in b.value.decode().split("\\n") if x and name in x]

def empty_cache(ctx):
    fake.fake_fail_alloc(0, 2)
    assert error(core.Tensor.create, ctx, (0, 0), [[(0, 0)]], [[1 << 28]]) == 2
    fake.fake_fail_alloc(0, 0)

def error(f, *a):
    try:
        f(*a)
    except MpsxxError as e:
        return e.code
    return 0
"""


@functools.lru_cache(maxsize=None)
def _fake() -> str:
    import __graft_entry__

    __graft_entry__.build()
    out = Path(tempfile.mkdtemp(prefix="fakecuda")) / "libfakecuda.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    "-I" + str(ROOT / "mpsxx_gb300" / "csrc"), str(ROOT / "tests" / "fake_cuda.cpp"), "-o", str(out)],
                   check=True)
    return str(out)


def run(code: str):
    """The JSON value that `code` leaves in `out`."""
    fake = _fake()
    text = PRELUDE.format(root=str(ROOT), fake=fake) + textwrap.dedent(code) + "\nprint('OUT' + json.dumps(out))\n"
    p = subprocess.run([sys.executable, "-c", text], capture_output=True, text=True, cwd=ROOT,
                       env=dict(os.environ, LD_PRELOAD=fake), timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
    return json.loads(p.stdout.split("OUT")[-1])


def operands(core, ctx, dims=(40, 24), nw=3, qrow=None, cols=None):
    """L, R and psi of a bond with the given row sector dimensions, without values; blocks
    without elements are stored as well."""
    n = len(dims)
    qa = qrow or [(i, 0) for i in range(n)]
    qb = [(n - a, 0) for a, _ in qa]
    qw = [(0, 0)] + [(s * k, 0) for k in range(1, nw) for s in (1, -1)]
    neg = lambda q: [(-x, -y) for x, y in q]  # noqa: E731
    d, e, one = list(dims), list(cols or dims), [1] * len(qw)

    def tensor(q, qs, ds):
        tags = [np.ravel_multi_index(i, [len(x) for x in qs]) for i in np.ndindex(*[len(x) for x in qs])
                if all(sum(x[k][c] for x, k in zip(qs, i)) == q[c] for c in range(2))]
        return core.Tensor.create(ctx, q, qs, ds, [int(t) for t in tags])

    return (tensor((0, 0), [qa, qw, neg(qa)], [d, one, d]), tensor((0, 0), [qb, neg(qw), neg(qb)], [e, one, e]),
            tensor((n, 0), [qa, qb], [d, e]))
