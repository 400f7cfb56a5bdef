"""Memory of large results: what is kept of dropped ones (CPU), and that an array's ids are its own whatever becomes of it (GPU)."""
import ctypes
import os
import signal
import subprocess

import numpy as np
import pytest

from conftest import ROOT, tiny_vocab

MB = 1 << 20


@pytest.fixture()
def memory(tmp_path):
    src = tmp_path / "wrap.cc"
    src.write_text('#include "result_memory.h"\n'
                   'extern "C" void* get(size_t n) { return result_memory::get(n); }\n'
                   'extern "C" void put(void* p) { result_memory::put(p); }\n'
                   'extern "C" void users(int c) { result_memory::users(c); }\n'
                   'extern "C" size_t kept_bytes() { return result_memory::kept().bytes; }\n'
                   'extern "C" int kept_count() { return result_memory::kept().n; }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "graphtok_b200", "pyhost"), "-o", str(tmp_path / "wrap.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(tmp_path / "wrap.so"))
    lib.get.restype, lib.get.argtypes, lib.put.argtypes = ctypes.c_void_p, [ctypes.c_size_t], [ctypes.c_void_p]
    lib.kept_bytes.restype = ctypes.c_size_t
    return lib


def test_kept_memory_is_bounded_and_given_back(memory):
    memory.put(memory.get(MB))
    assert memory.kept_count() == 0                  # no tokenizer is open
    memory.users(1)
    a = memory.get(10 * MB)
    memory.put(a)
    assert memory.kept_count() == 1
    assert memory.get(10 * MB + 100000) == a         # about the same size
    assert memory.kept_count() == 0
    memory.put(a)
    small = memory.get(MB)
    assert small != a                                # far too large for that
    for size in (300 << 20, 100 << 10):              # beyond the bound, and left to malloc
        memory.put(memory.get(size))
        assert memory.kept_count() == 1
    blocks = [memory.get(s * MB) for s in (3, 5, 9, 90, 90, 90)]
    for b in blocks + [small]:
        memory.put(b)
        assert memory.kept_count() <= 4 and memory.kept_bytes() <= 256 * MB
    memory.users(1)
    memory.users(-1)
    assert memory.kept_count() > 0
    memory.users(-1)
    assert memory.kept_count() == 0 and memory.kept_bytes() == 0


@pytest.fixture(scope="module")
def tok():
    from graphtok_b200.gpu_bpe_tokenizer import Tokenizer
    return Tokenizer(tiny_vocab("llama3"))


def large(k):
    """Texts of some 400,000 ids (1.6 MB of them)."""
    return ("%d " % k + "many words of one kind or another, " * 24000).encode()


@pytest.mark.gpu
def test_large_results_own_their_memory(tok, oracles):
    want = oracles["llama3"].encode(large(1))
    for ids in (tok.encode_numpy(large(1)), tok.encode_batch([large(1)])[0], tok._g.encode_batch(large(1), [0, len(large(1))])[0]):
        assert ids.flags.owndata and ids.flags.writeable and np.array_equal(ids, want) and ids.nbytes > MB
        ids.resize(3 * want.size, refcheck=False)
        assert np.array_equal(ids[:want.size], want) and not ids[want.size:].any()


@pytest.mark.gpu
def test_an_upload_of_a_dropped_result(tok, oracles):
    """An asynchronous copy of a result to the device, the result dropped before the copy has run."""
    import torch
    want = oracles["llama3"].encode(large(2))
    ids = tok.encode_numpy(large(2))
    tok.encode_numpy(large(3))
    torch.cuda._sleep(200_000_000)
    up = torch.from_numpy(ids.view(np.int32)).to("cuda", non_blocking=True)
    del ids
    for k in range(4, 8):
        tok.encode_numpy(large(k))
    assert np.array_equal(up.cpu().numpy().view(np.uint32), want)


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:This process .* is multi-threaded")
def test_a_result_in_a_forked_child(tok, oracles):
    """A child that holds a result which its parent has dropped since: still the child's own."""
    want = oracles["llama3"].encode(large(8))
    ids = tok.encode_numpy(large(8))
    read, write = os.pipe()
    child = os.fork()
    if child == 0:
        signal.alarm(20)
        os.read(read, 1)
        os._exit(0 if np.array_equal(ids, want) else 1)
    del ids
    for k in range(9, 13):
        tok.encode_numpy(large(k))
    os.write(write, b"x")
    assert os.waitstatus_to_exitcode(os.waitpid(child, 0)[1]) == 0
