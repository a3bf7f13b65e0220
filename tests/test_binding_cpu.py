"""The CPython binding's argument conversion, without a GPU: what it cannot convert raises in Python, as Tensor.data_ptr() and
ctypes do, and never ends the process (so the calls run in a child)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRELUDE = """
import ctypes, torch
import helios_glm53flash_b200 as hk
from helios_glm53flash_b200 import _binding as nb
lib = hk.load_library()
nb.bind({n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in hk.SIGNATURES})
class stream: cuda_stream = 0
t = torch.zeros(4)
def gate(b=t, f=t, lb=-5.0, beta=t, S=0, stream=stream):        # S = 0: returns before any launch
    return nb.hk_kda_gate(b, f, t, t, lb, beta, t, S, 1, 1, stream)
def raises(kind, fn):
    try:
        fn()
    except kind as e:
        print("raised", type(e).__name__, e)
    else:
        raise SystemExit("no " + kind.__name__)
assert gate() == hk.HK_OK
"""


def _child(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, "exit %d\n%s\n%s" % (r.returncode, r.stdout, r.stderr[-2000:])


@pytest.fixture(scope="module", autouse=True)
def built():
    from helios_glm53flash_b200 import build as hk_build
    return hk_build.build()


@pytest.mark.parametrize("body", [
    "raises(RuntimeError, lambda: gate(b=torch.eye(3).to_sparse()))",                        # no storage
    "raises(RuntimeError, lambda: torch.func.vmap(lambda x: (gate(beta=x), x)[1])(torch.zeros(2, 3)))",
])
def test_a_tensor_without_an_address_raises(body):
    _child(body)


def test_arguments_of_the_wrong_kind_raise():
    _child("""
raises(AttributeError, lambda: gate(b=3))
raises(TypeError, lambda: gate(S=1.5))
raises(TypeError, lambda: gate(S=2 ** 40))
raises(TypeError, lambda: gate(lb="x"))
raises(AttributeError, lambda: gate(stream=7))
raises(TypeError, lambda: nb.hk_kda_gate(t, t))
raises(TypeError, lambda: nb.hk_gated_rms_norm(t, t, t.int(), t, t, t, t, 0, 4, 1e-6, 0.0, 1, 0, 0, stream))     # dtype tag
""")


def test_lazily_cloned_tensors_get_their_own_memory_only_where_they_are_written():
    _child("""
a, b = t._lazy_clone(), t._lazy_clone()
gate(b=a, beta=b)
assert torch._C._is_cow_tensor(a) and not torch._C._is_cow_tensor(b)
""")
