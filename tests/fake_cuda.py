"""Runs a channel's host code without a GPU, on the stand-in runtime of tests/fake_cudart.c, and
reads its log."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def build(tmp):
    so = str(tmp / "libfake_cudart.so")
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-Wall", "-Werror", "-fPIC", "-shared",
                    os.path.join(HERE, "fake_cudart.c"), "-o", so], check=True)
    return so


def run(so, log, code, args=""):
    """Runs `code` in a process of its own; returns (its standard output, the log's lines as lists)"""
    env = dict(os.environ, LD_PRELOAD=so, FAKE_CUDART_LOG=str(log), FAKE_CUDART_ARGS=args, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return r.stdout, [l.split() for l in open(log)]


def allocations(lines):
    """[(first byte, bytes)] of the device arrays"""
    return [(int(l[1], 16), int(l[2])) for l in lines if l[0] == "A"]


def launches(lines, kernel):
    """[(position in the log, grid, [arguments])] of the launches whose name contains `kernel`"""
    return [(i, tuple(int(x) for x in l[3:6]), [0 if x == "(nil)" else int(x, 16) for x in l[10:]])
            for i, l in enumerate(lines) if l[0] == "L" and kernel in l[1]]


def concurrent(lines, kernel):
    """The kernels that no stream order or event orders against a launch whose name contains `kernel`"""
    on, at, before = {}, {}, []  # launches that a stream's next one / an event's waiters follow; per launch
    names = []
    for l in lines:
        if l[0] == "L":
            names.append(l[1])
            before.append(frozenset(on.get(l[2], ())))
            on[l[2]] = before[-1] | {len(names) - 1}
        elif l[0] == "R":
            at[l[1]] = on.get(l[2], frozenset())
        elif l[0] == "W":
            on[l[1]] = on.get(l[1], frozenset()) | at.get(l[2], frozenset())
    mine = [i for i, n in enumerate(names) if kernel in n]
    return mine, {names[j] for i in mine for j in range(len(names)) if j != i and j not in before[i] and i not in before[j]}
