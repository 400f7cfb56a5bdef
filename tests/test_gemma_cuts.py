"""Cuts of the Gemma-3 shape, where the bit planes can go wrong: whole, broken and unknown characters, U+2581 and spaces, added
tokens and document starts, moved byte by byte over a chunk's, a mask word's and a tile's edge.  Against the oracle, which does not cut."""
import random

import numpy as np
import pytest

TILE = 8000          # bytes of text per pre-tokenization tile
PIECES = [b" ", b"  ", b"a", b"the", b" of", "▁".encode(), "▁▁".encode(), "é".encode(), "中".encode(), "\U0001F600".encode(), "ก".encode(),
          b"\x80", b"\xE2\x96", b"\xE2", b"\xC3", b"\xF0\x9F\x98", b"\xED\xA0\x80", b"\xC0\xAF", b"\xE0\x80\x80", b"\xF4\x90\x80\x80", b"\xFF", b"\x81 ", b"\n", b"\t",
          b"<bos>", b"<bo", b"\xE2<bos>\x96\x81", b"\x00", b"~", b"Zq"]


def mixture(rng, count):
    return b"".join(rng.choice(PIECES) for _ in range(count))


@pytest.mark.parametrize("edge", (16, 32, 128, TILE, 2 * TILE))
def test_pieces_across_an_edge(emuls, oracles, edge):
    rng = random.Random(edge)
    e, o = emuls["gemma"], oracles["gemma"]
    for shift in range(-9, 3):
        text = (b"ab " * edge)[:edge + shift] + mixture(rng, 60)
        want = o.encode_normalized(text)
        for reverse in (False, True):
            assert np.array_equal(e.encode(text, reverse=reverse), want), (shift, text[edge + shift:])


def test_mixtures_and_document_starts(emuls, oracles):
    rng = random.Random(7)
    e, o = emuls["gemma"], oracles["gemma"]
    for _ in range(150):
        text = mixture(rng, rng.randint(1, 90))
        assert np.array_equal(e.encode(text), o.encode_normalized(text)), text
        # the same bytes cut into documents anywhere, inside characters too: each document as if it were alone
        cuts = sorted(rng.randint(0, len(text)) for _ in range(rng.randint(0, 6)))
        offsets = np.array([0] + cuts + [len(text)], dtype=np.uint32)
        ids, doc = e.encode(text, offsets=offsets)
        parts = [o.encode_normalized(text[int(a):int(b)]) for a, b in zip(offsets[:-1], offsets[1:])]
        assert np.array_equal(ids, np.concatenate(parts)), (text, cuts)
        assert doc.tolist() == [0] + np.cumsum([len(p) for p in parts]).tolist()
