"""The CPython extension by itself (no GPU): what it does with its arguments before and while the library works, the library's
calls stood in for by functions of the test where they are reached.  Each test in a process of its own."""
import numpy as np
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
for call in (lambda: host.encode_batch(0, texts, False), lambda: host.encode_to_device(0, texts, False, None, None)):
    try:
        call()
    except MemoryError:
        print("refused", end=" ")
""") == "refused refused"


def test_a_buffer_that_changes_during_the_call(built):
    """A bytearray, alone, in a batch and under a view: its bytes of before the call, and free to be resized meanwhile."""
    assert extension("""
seen = []
def measure(handle, pieces, n, batch):
    buf.extend(b"more" * 100)                            # BufferError while somebody holds the buffer
    buf[:5] = b"other"
    at, units = ctypes.c_void_p.from_address(pieces).value, ctypes.c_uint64.from_address(pieces + 8).value
    seen.append(ctypes.string_at(at, units))
    return -1
stand_in(measure=measure)
for form in (lambda b: host.encode(1, b, False), lambda b: host.encode_batch(1, (b,), False), lambda b: host.encode_to_device(1, b, False, None, None)):
    buf = bytearray(b"first and the rest")
    form(buf)
buf, whole = bytearray(b"another"), bytearray(b"under a view")
host.encode(1, memoryview(whole), False)
print(seen == [b"first and the rest"] * 3 + [b"under a view"], end="")
""") == "True"


def test_ids_of_other_types_in_gtok_decode():
    """GTok.decode converts to uint32 as numpy does, whatever takes the ids then (Tokenizer.decode checks their range first)."""
    from graphtok_b200 import GTok
    got = []

    class Host:
        def decode(self, handle, ids):
            got.append(ids)
            return b"text"
    g = GTok.__new__(GTok)
    g.handle, g.host = None, Host()
    for ids, want in (([1, 2], [1, 2]), (np.array([5, (1 << 32) + 6, -1]), [5, 6, 0xFFFFFFFF]), (np.array([7, -2], dtype=np.int32), [7, 0xFFFFFFFE]),
                      (np.array([3.0]), [3]), ((), [])):
        assert g.decode(ids) == b"text" and got[-1].dtype == np.uint32 and got[-1].tolist() == want
    for bad in ([-1], [1 << 32]):
        with pytest.raises(OverflowError):
            g.decode(bad)


def test_staging_on_a_closed_handle():
    """The library answers no cap for a closed handle: an error, not an endless search for a cap that is large enough."""
    assert child("""
import faulthandler
faulthandler.dump_traceback_later(20, exit=True)
from graphtok_b200 import GTok, GTokError, load_lib
from graphtok_b200.gpu_bpe_tokenizer import Tokenizer
t = Tokenizer.__new__(Tokenizer)
t._g = GTok.__new__(GTok)
t._g.lib, t._g.handle = load_lib(), None
for call in (lambda: t.bench_stage("text"), lambda: t.bench_stage_batch(["text"])):
    try:
        call()
    except GTokError:
        print("refused", end=" ")
""").split() == ["refused"] * 2


def test_a_list_that_changes_while_decoding_makes_its_buffers(built):
    """The buffers are made with the interpreter lock let go: a list that is another one afterwards goes the caller's other way."""
    assert extension("""
room = (ctypes.c_uint32 * 100000)()
def decode_room(handle, n):
    change()
    return ctypes.addressof(room)
stand_in(decode_room=decode_room)
for change in (lambda: ids.clear(), lambda: ids.append(1), lambda: ids.__setitem__(99999, "x")):
    ids = [1 << 20] * 100000
    print(host.decode(1, ids), end=" ")
""") == "None None None"
