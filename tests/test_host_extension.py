"""The host extension (csrc/fo_host.cc) where it needs no GPU: walks over trees that it hands back to the Python walk (their
leaves are no CUDA tensors) or that it has to refuse, and the bookkeeping of compiled step plans around it."""

import time

import pytest
import torch

from flashoptim_jax_b200 import _engine as eng
from flashoptim_jax_b200 import _lib


def test_trees_are_compiled_in_linear_time():
    """set_fp32_params compiles the tree on every call: 16 times the keys may take 16 times as long (64 allows for the sort and the
    cache), not 256 times."""
    host = _lib.host()

    def best(n):
        tree = {f"{i * 7919 % n:06d}": None for i in range(n)}  # inserted out of order
        times = []
        for _ in range(5):
            t = time.perf_counter()
            assert host.split(tree, tree, 8) is None
            times.append(time.perf_counter() - t)
        return min(times)

    best(100)
    assert best(32000) < 64 * best(2000)


def test_plans_reordered_by_another_thread_do_not_lose_a_step():
    """While one thread's step runs on the second plan, another moves that plan to the front or drops plans."""
    native = eng.NativeStep(_lib.FO_OPT_ADAM, True, {}, None, None)
    miss = lambda *a: None

    def run(*a):
        native.plans = type(native.plans)(native.plans[1:2])  # what the other thread does meanwhile
        return "the step"

    native.plans = type(native.plans)([(miss, 0), (miss, 1), (run, 2)])
    assert native.run(None, None, (), None) == "the step"
    assert (run, 2) in native.plans


def test_trees_without_an_end_are_a_recursion_error():
    """In a process of its own: without the check the stack runs out."""
    import os
    import subprocess
    import sys

    code = """
from flashoptim_jax_b200 import _lib
h = _lib.host()
a = []; a.append(a)
b = {}; b["x"] = (b,)
deep = None
for _ in range(200000): deep = [deep]
for tree in (a, b, deep):
    for call in (lambda: h.sq_norm(tree), lambda: h.reconstruct(tree, tree), lambda: h.split(tree, tree, 8)):
        try:
            call()
            raise SystemExit("accepted")
        except RecursionError:
            pass
while deep is not None: deep = deep[0]
print("refused")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "refused", (r.returncode, r.stderr[-500:])


def test_keys_of_mixed_types_go_to_the_python_walk():
    """Keys whose comparison is code of the user's, behind a key that is out of order."""

    class Key:
        def __lt__(self, other):
            tree.clear()
            return True

        __gt__ = __lt__

    tree = {"b": None, "a": None, Key(): None}
    assert _lib.host().sq_norm(tree) is None
    assert len(tree) == 3
