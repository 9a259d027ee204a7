"""Host layouts where the host runs out of threads or memory: the call ends in its result or in
PRISM_ERR_ALLOC, never in an aborted process.  Each limit on the address space is set in a
process of its own: the lowest leave no room for a thread's stack, the others run out of memory
at one place or another, in the caller's thread or in one of the layout's."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

CHILD = r"""
import os, resource, sys
import numpy as np
import prispack_b200 as P
P.load()
n = int(sys.argv[2])
rng = np.random.default_rng(0)
# five entries a row among the rows before it, some of them far away
dep = [np.unique(np.maximum(i - rng.integers(1, 400, 5), 0)) if i else np.zeros(0, int) for i in range(n)]
rp = np.concatenate([[0], np.cumsum([len(d) for d in dep])]).astype(np.uint32)
ci = np.concatenate(dep).astype(np.uint32)
v, b = np.full(len(ci), 0.1), np.ones(n)
del dep
call = {"flow": lambda: P.selftest_flow_layout(rp, ci, v, b, num_slabs=40),
        "rounds": lambda: P.selftest_stream_layout(rp, ci, v, b, num_ctas=40, rows_per_cta=0)}[sys.argv[1]]
want = call()
for extra in range(1, 40, 3):  # MB beyond what the process has mapped
    pid = os.fork()
    if pid == 0:
        used = int(open("/proc/self/statm").read().split()[0]) * os.sysconf("SC_PAGE_SIZE")
        resource.setrlimit(resource.RLIMIT_AS, (used + (extra << 20), used + (extra << 20)))
        try:
            rc = 0 if np.array_equal(call(), want) else 3
        except P.PrismError as e:
            rc = 0 if e.status == 8 else 4
        except MemoryError:
            rc = 0
        os._exit(rc)
    status = os.waitpid(pid, 0)[1]
    if status != 0:
        print(f"{extra} MB: wait status {status:#x}")
        sys.exit(1)
"""


@pytest.mark.parametrize("layout", ["flow", "rounds"])
def test_a_host_out_of_threads_or_memory(layout):
    env = dict(os.environ, PRISM_LAYOUT_THREADS="6", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, layout, "40000"], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
