"""What the extension `_host` does, by ctypes alone: for an installation without it (no Python or numpy headers
where it was built, or an interpreter it was not built for).

The same four functions with the same arguments and answers, over the calls of gtok.h that take one run of
bytes: a str is encoded by the interpreter and a batch is joined first, which the extension does without.
"""
import ctypes

import numpy as np

MOST_BYTES = 0xFFFFFF00          # beyond it a length does not fit the calls; they answer -3 for longer texts


def as_bytes(text):
    if isinstance(text, str):
        return text.encode("utf-8")
    if isinstance(text, (bytes, bytearray, memoryview)):
        return bytes(text)
    raise TypeError("text must be str or bytes")


def concatenated(texts):
    """(bytes, n + 1 offsets) of a sequence of texts; offsets None where they do not fit 32 bits."""
    blobs = [as_bytes(t) for t in texts]
    ends = np.cumsum([len(b) for b in blobs], dtype=np.int64)
    if ends[-1] > MOST_BYTES:
        return b"", None
    offsets = np.zeros(len(blobs) + 1, dtype=np.uint32)
    offsets[1:] = ends
    return b"".join(blobs), offsets


class CtypesHost:
    """`lib`: libgtok.so as load_lib() returns it."""

    def __init__(self, lib):
        self.lib = lib

    def users(self, change):
        pass                     # nothing is kept between calls

    def _grow(self, handle, n_bytes):
        # doubled until a text of that many bytes fits even if NFC lengthens it (at most threefold)
        cap = int(self.lib.gtok_x_set_max_bytes(handle, 0))
        need = 3 * n_bytes + 64
        if not cap or cap >= need:
            return
        while cap < need:
            cap *= 2
        self.lib.gtok_x_set_max_bytes(handle, min(cap, 0xFFFFFFFF))

    def encode(self, handle, text, grow):
        data = as_bytes(text)
        if len(data) > MOST_BYTES:
            return -3
        if grow:
            self._grow(handle, len(data))
        for room in (len(data) + 16, 3 * len(data) + 64):      # (more ids than bytes: only text that NFC lengthens)
            out = np.empty(room, dtype=np.uint32)
            n = self.lib.gtok_encode(handle, data, len(data), out.ctypes.data, min(room, 0xFFFFFFFF))
            if n != -2:
                break
        return n if n < 0 else out[:n].copy()

    def encode_batch(self, handle, texts, grow):
        blob, offsets = concatenated(texts)
        if offsets is None:
            return -3
        if grow:
            self._grow(handle, len(blob))
        doc = np.empty(offsets.size, dtype=np.uint32)
        for room in (len(blob) + 16, 3 * len(blob) + 64):
            out = np.empty(room, dtype=np.uint32)
            n = self.lib.gtok_encode_batch(handle, blob, offsets.ctypes.data, offsets.size - 1, out.ctypes.data, min(room, 0xFFFFFFFF), doc.ctypes.data)
            if n != -2:
                break
        return n if n < 0 else (out[:n].copy(), doc)

    def encode_to_device(self, handle, text, grow, make, queue):
        batch = text.__class__ is tuple
        if batch:
            blob, offsets = concatenated(text)
            if offsets is None:
                return -3
        else:
            blob = as_bytes(text)
            if len(blob) > MOST_BYTES:
                return -3
        if grow:
            self._grow(handle, len(blob))
        doc = make(offsets.size) if batch else None
        for room in (len(blob) + 16, 3 * len(blob) + 64):
            out = make(room)
            if self.lib.gtok_x_result_stream(handle, queue()) < 0:
                return -1
            at, most = ctypes.c_void_p(out.data_ptr()), min(room, 0xFFFFFFFF)
            if batch:
                n = self.lib.gtok_x_encode_batch_to_device(handle, blob, offsets.ctypes.data, offsets.size - 1, at, most, ctypes.c_void_p(doc.data_ptr()))
            else:
                n = self.lib.gtok_encode_to_device(handle, blob, len(blob), at, most)
            if n != -2:
                break
        return n if n < 0 else (out, n, doc)

    def decode(self, handle, ids):
        return None              # the caller goes by an array, as for an `ids` that the extension does not take
