"""The CPython extension by itself (no GPU): what it does with its arguments before and while the library works, the library's
calls stood in for by functions of the test where they are reached.  Each test in a process of its own."""
import pytest

from test_build_and_load import child

HEAD = """
import ctypes, resource, sys
from graphtok_b200 import load_lib
host = load_lib().host
if type(host).__name__ == "CtypesHost":
    print("no extension")
    sys.exit()
made = {}
def stand_in(**calls):
    for name, f in calls.items():
        made["gtok_x_" + name] = ctypes.CFUNCTYPE(ctypes.c_int64, *[ctypes.c_void_p] * f.__code__.co_argcount)(f)
    lib = load_lib()
    host.bind(lambda name: ctypes.cast(made.get(name) or getattr(lib, name), ctypes.c_void_p).value)
"""


def extension(code):
    out = child(HEAD + code).strip()
    if out == "no extension":
        pytest.skip("the extension is not built here")
    return out


def test_no_memory_for_a_calls_notes(built):
    """An allocation of the extension's own that fails is a MemoryError, not the end of the process."""
    assert extension("""
texts = ("a",) * 20_000_000
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (100 << 20),) * 2)
for call in (lambda: host.encode_batch(0, texts, False), lambda: host.encode_to_device(0, texts, False, None)):
    try:
        call()
    except MemoryError:
        print("refused", end=" ")
""") == "refused refused"
