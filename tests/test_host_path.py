"""The way of Python objects to the library and back: UTF-8 form of a str's characters (CPU), and the calls of
gpu_bpe_tokenizer that take text and ids as Python holds them (GPU), each against the interpreter's own UTF-8
form encoded by the same handle from one bytes object, or against the oracle."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

from conftest import ROOT, tiny_vocab

WIDTH = {"ascii": (0x20, 0x7E), "latin1": (0xA0, 0xFF), "ucs2": (0x400, 0xD7FF), "ucs4": (0x1F300, 0x1F5FF)}


def _text(kind, n, seed):
    rng = random.Random("%s %d %d" % (kind, n, seed))
    lo, hi = WIDTH[kind]
    out = [chr(rng.randint(lo, hi)) if rng.random() < 0.4 else chr(rng.choice((32, 97, 101, 110, 116, 10))) for _ in range(n)]
    if n:
        out[rng.randrange(n)] = chr(hi)        # the str has the width its kind stands for
    return "".join(out)


@pytest.fixture(scope="module")
def utf8(tmp_path_factory):
    d = tmp_path_factory.mktemp("utf8")
    src = d / "wrap.cc"
    src.write_text('#include "host_text.h"\n'
                   'extern "C" unsigned long long size(const void* p, unsigned long long n, unsigned k) { return gtok::utf8_size(p, n, k); }\n'
                   'extern "C" unsigned long long put(unsigned char* d, const void* p, unsigned long long n, unsigned k) { return gtok::utf8_write(d, p, n, k) - d; }\n'
                   'extern "C" unsigned long long stream(unsigned char* d, const void* p, unsigned long long n, unsigned k) { return gtok::utf8_stream(d, p, n, k) - d; }\n')
    csrc = os.path.join(ROOT, "graphtok_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O3", "-fPIC", "-shared", "-I" + csrc, "-o", str(d / "wrap.so"), str(src), os.path.join(csrc, "host_text.cc")], check=True)
    lib = ctypes.CDLL(str(d / "wrap.so"))
    lib.size.restype = lib.put.restype = lib.stream.restype = ctypes.c_ulonglong
    lib.size.argtypes = [ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_uint]
    lib.put.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_uint]
    lib.stream.argtypes = lib.put.argtypes
    return lib


@pytest.mark.parametrize("width,kind", [(1, 3), (2, 2), (4, 4)])
@pytest.mark.parametrize("n", [0, 1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 79, 80, 127, 128, 129, 1000, 1025, 3000])
def test_utf8_form(utf8, width, kind, n):
    """Every length class of characters at the edges of the 16-, 32- and 64-character steps; nothing written past the end."""
    rng = np.random.default_rng(n * 8 + width)
    top = {1: 0xFF, 2: 0xFFFF, 4: 0x10FFFF}[width]
    for mode in range(6):
        limit = [0x7F, 0x80, 0x7FF, 0x800, 0xFFFF, top][mode]
        cps = rng.integers(0, min(limit, top) + 1, n)
        cps[(cps >= 0xD800) & (cps < 0xE000)] = 0xE000 if top > 0xFF else 0x41
        units = cps.astype({1: np.uint8, 2: np.uint16, 4: np.uint32}[width])
        want = "".join(map(chr, cps)).encode("utf-8")
        assert utf8.size(units.ctypes.data, n, kind) == len(want)
        out = np.full(len(want) + 80, 0xAA, dtype=np.uint8)
        assert utf8.put(out.ctypes.data, units.ctypes.data, n, kind) == len(want)
        assert out[:len(want)].tobytes() == want and (out[len(want):] == 0xAA).all()
        for at in (0, 1, 63, 64):                # wherever in a line the destination begins
            out = np.full(at + len(want) + 80, 0xAA, dtype=np.uint8)
            assert utf8.stream(out.ctypes.data + at, units.ctypes.data, n, kind) == len(want)
            assert out[at:at + len(want)].tobytes() == want and (out[:at] == 0xAA).all() and (out[at + len(want):] == 0xAA).all()
        if n and width > 1:
            units[n // 2] = 0xDC00
            assert utf8.size(units.ctypes.data, n, kind) == 0xFFFFFFFFFFFFFFFF


def _tokenizer(family, route):
    """A tokenizer that goes by the extension, or one that goes by ctypes as where the extension was not built."""
    from graphtok_b200.ctypes_host import CtypesHost
    from graphtok_b200.gpu_bpe_tokenizer import Tokenizer
    t = Tokenizer(tiny_vocab(family))
    if route == "ctypes":
        t._host = t._g.host = CtypesHost(t._g.lib)
    elif isinstance(t._host, CtypesHost):
        pytest.skip("the extension is not built here")
    return t


@pytest.fixture(scope="module", params=["extension", "ctypes"])
def tok(request):
    return _tokenizer("llama3", request.param)


# sizes: single-block route and its limit, one copy step and several, the size from which characters are shared among
# threads, results below and above the size from which the memory of dropped ones is kept
@pytest.mark.gpu
@pytest.mark.parametrize("kind", list(WIDTH))
@pytest.mark.parametrize("n", [0, 1, 33, 2047, 2049, 40000, 70001, 400003])
def test_str_and_bytes_alike(tok, oracles, kind, n):
    text = _text(kind, n, 1)
    data = text.encode("utf-8")
    want = oracles["llama3"].encode(data)
    for form in (text, data, bytearray(data), memoryview(data), memoryview(data[::-1])[::-1]):
        got = tok.encode_numpy(form)
        assert got.dtype == np.uint32 and got.flags.writeable and np.array_equal(got, want)
    assert np.array_equal(tok.encode_to_device(text).cpu().numpy(), want)
    assert tok.decode_bytes(want) == tok._g.decode(want.astype(np.int64)) == data


@pytest.mark.gpu
@pytest.mark.parametrize("docs,longest", [(1, 50), (7, 0), (300, 40), (40, 30000), (3, 300000)])
def test_batch_of_mixed_objects(tok, oracles, docs, longest):
    rng = random.Random(docs)
    texts = [_text(rng.choice(list(WIDTH)), rng.randint(0, longest), i) for i in range(docs)]
    form = (lambda s: s, lambda s: s.encode(), lambda s: bytearray(s.encode()), lambda s: memoryview(s.encode()))
    ids, off = tok.encode_batch(form[i % 4](s) for i, s in enumerate(texts))
    want = [oracles["llama3"].encode(s.encode()) for s in texts]
    assert off.tolist() == np.concatenate([[0], np.cumsum([w.size for w in want])]).tolist()
    assert np.array_equal(ids, np.concatenate(want))
    dev, dev_off = tok.encode_batch_to_device(texts)
    assert np.array_equal(dev.cpu().numpy(), ids.astype(np.int32)) and dev_off.cpu().tolist() == off.tolist()


NFC_TEXTS = {
    "nothing to do": "plain words " * 40,
    "composed": "Cafe\u0301 a\u0323\u0302 " * 60,
    "growing": "\u0958\u0959 \U0001d15e" * 300,                      # more bytes than before, and more ids than there were bytes
    "a stretch too long for the device": "q" + "\u0301\u0323" * 150 + " \u0958" * 50,
    "empty": "",
}


@pytest.mark.gpu
@pytest.mark.parametrize("route", ("extension", "ctypes"))
def test_texts_that_normalisation_changes(oracles, route):
    """The vocabulary that declares NFC: each text alone, as part of a batch, to the host and to the device."""
    tok, o = _tokenizer("qwen25", route), oracles["qwen25"]
    want = {k: o.encode(t.encode()) for k, t in NFC_TEXTS.items()}
    assert want["growing"].size > len(NFC_TEXTS["growing"].encode())
    for repeat in (1, 40):
        for name, text in NFC_TEXTS.items():
            text = text * repeat
            expect = o.encode(text.encode()) if repeat > 1 else want[name]
            assert np.array_equal(tok.encode_numpy(text), expect), name
            assert np.array_equal(tok.encode_numpy(text.encode()), expect), name
            assert np.array_equal(tok.encode_to_device(text).cpu().numpy(), expect), name
    names = list(NFC_TEXTS) * 30
    for chosen in (names, ["growing"] * 3, ["empty", "growing"], ["nothing to do"] * 5):
        texts = [NFC_TEXTS[n] if i % 2 else NFC_TEXTS[n].encode() for i, n in enumerate(chosen)]
        ids, off = tok.encode_batch(texts)
        assert np.array_equal(ids, np.concatenate([want[n] for n in chosen])), chosen[:3]
        assert off.tolist() == [0] + np.cumsum([want[n].size for n in chosen]).tolist()
        dev, dev_off = tok.encode_batch_to_device(texts)
        assert np.array_equal(dev.cpu().numpy(), ids.astype(np.int32)) and dev_off.cpu().tolist() == off.tolist()


@pytest.mark.gpu
def test_normalised_text_beyond_the_byte_cap(oracles):
    """A text within the handle's cap whose normalised form is not: refused, and encoded once the cap is raised."""
    from graphtok_b200 import GTok, GTokError
    text = (NFC_TEXTS["growing"] * 2).encode()
    for raise_to in (3 * len(text), 8 * len(text)):
        g = GTok(tiny_vocab("qwen25"), max_bytes=len(text))
        with pytest.raises(GTokError, match="-3"):
            g.encode(text)
        g.set_max_bytes(raise_to)
        assert np.array_equal(g.encode(text), oracles["qwen25"].encode(text))
        g.close()


@pytest.mark.gpu
def test_results_outlive_later_calls(tok, oracles):
    """Large results held at once, and a view of a dropped one: each stays as it was."""
    texts = [_text("ucs2", 120000, i) for i in range(9)]
    got = [tok.encode_numpy(t) for t in texts]
    for t, g in zip(texts, got):
        assert np.array_equal(g, oracles["llama3"].encode(t.encode()))
    part = got[0][5:9]
    keep = part.tolist()
    del got
    tok.encode_numpy(texts[8])
    assert part.tolist() == keep


@pytest.mark.gpu
@pytest.mark.parametrize("side_stream", (False, True))
@pytest.mark.parametrize("texts", ("one", "batch", "batch without text"))
def test_results_on_the_device_wait_for_the_readers_of_their_memory(tok, oracles, side_stream, texts):
    """A tensor dropped while work that reads it is still queued: the ids that get its block come after that work."""
    import torch
    text = _text("ucs2", 3000, 4)
    want = oracles["llama3"].encode(text.encode())
    encode = {"one": lambda: (tok.encode_to_device(text), want), "batch": lambda: (tok.encode_batch_to_device([text, ""])[0], want),
              "batch without text": lambda: (tok.encode_batch_to_device(["", "", ""])[1], np.zeros(4))}[texts]
    encode()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()                              # so that the block dropped below is the smallest one that fits
    with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.current_stream()):
        held = torch.full((32768,), 7, dtype=torch.int32, device="cuda")
        at = held.data_ptr()
        torch.cuda._sleep(200_000_000)                    # some 0.1 s
        seen = held + 1
        del held
        got, expect = encode()
        assert at <= got.data_ptr() < at + 4 * 32768      # the block has come back, as the test wants it to
        assert (seen.cpu() == 8).all() and np.array_equal(got.cpu().numpy(), expect)


@pytest.mark.gpu
def test_refused_inputs(tok):
    for bad in (3, None, [1], ("a",)):
        with pytest.raises(TypeError):
            tok.encode_numpy(bad)
        with pytest.raises(TypeError):
            tok.encode_batch(["a", bad])
        with pytest.raises(TypeError):
            tok.encode_to_device(bad)
    for lone in ("\ud800", "a" * 100 + "\udfff" + "b" * 100, "\U0001F600\udc00"):
        with pytest.raises(UnicodeEncodeError):
            tok.encode_numpy(lone)
        with pytest.raises(UnicodeEncodeError):
            tok.encode_batch(["fine", lone])
    for bad in ([5, -1], [1 << 32], np.array([-1], dtype=np.int32), np.array([1 << 32]), np.array([1 << 32], dtype=np.uint64)):
        with pytest.raises(ValueError):
            tok.decode_bytes(bad)
    for ids in ([72, 105], [True, 3], np.array([[72, 105]], dtype=np.uint16), np.arange(40)[::2], np.arange(9, dtype=np.int32), (7, 8), []):
        assert tok.decode_bytes(ids) == tok._g.decode(np.asarray(ids).astype(np.uint32).reshape(-1), want_ms=True)[0]
    assert tok.encode_numpy("still works").size > 0


class Piece(ctypes.Structure):
    _fields_ = [("data", ctypes.c_void_p), ("units", ctypes.c_uint64), ("kind", ctypes.c_uint32)]


@pytest.mark.gpu
def test_steps_out_of_order_are_refused(oracles):
    """gtok_x_measure, gtok_x_encode_measured, gtok_x_take_ids: a length that was not measured, a step twice, a step whose call
    another one has ended."""
    from graphtok_b200 import GTok
    g = GTok(tiny_vocab("llama3"))
    lib, h = g.lib, ctypes.c_void_p(g.handle)
    for name, types in (("gtok_x_measure", [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_int32]),
                        ("gtok_x_encode_measured", [ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p])):
        getattr(lib, name).restype, getattr(lib, name).argtypes = ctypes.c_int64, types
    lib.gtok_x_take_ids.restype, lib.gtok_x_take_ids.argtypes = ctypes.c_int32, [ctypes.c_void_p] * 3
    for size in (100, 50000):                    # the single-block route and the other
        text = _text("ascii", size, 9).encode()
        want = oracles["llama3"].encode(text)
        keep = ctypes.create_string_buffer(text)
        piece = Piece(ctypes.addressof(keep), len(text), 1)
        out = np.zeros(len(text) + 16, dtype=np.uint32)

        def measure():
            return lib.gtok_x_measure(h, ctypes.byref(piece), 1, 0)

        def encode(n):
            return lib.gtok_x_encode_measured(h, n, None, 0, None)

        def take():
            return lib.gtok_x_take_ids(h, out.ctypes.data, None)
        assert measure() == len(text)
        assert encode(len(text) - 1) == encode(len(text) + 1) == encode(0) == -1
        assert take() == -1                      # nothing encoded yet
        assert encode(len(text)) == want.size and encode(len(text)) == -1
        assert lib.gtok_x_take_ids(h, None, None) == -1
        assert take() == 0 and np.array_equal(out[:want.size], want) and take() == -1
        for other in (lambda: g.encode(b"other"), lambda: g.encode_batch(b"other", [0, 2, 5]), lambda: g.stage(b"other"), lambda: (g.stage(b"other"), g.replay())):
            assert measure() == len(text)
            other()
            assert encode(len(text)) == -1
            g.stage(b"first")
            assert measure() == len(text) and encode(len(text)) == want.size
            other()
            assert take() == -1
    assert "finished" in lib.gtok_x_last_error().decode()
    g.close()
