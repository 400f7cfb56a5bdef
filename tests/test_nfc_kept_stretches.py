"""The normalisation tile program keeps the normalised stretches of a 16-byte chunk from sizing to writing, up to eight of them,
28 bytes in all and 15 each: chunks at and beyond each limit, moved over a chunk's and a tile's edge, against unicodedata."""
import unicodedata

import pytest

import oracle_lib

TILE = 4096
STRETCHES = {
    "pairs": "éôạ" * 6,                      # composed, several a chunk
    "marks": "́ẍ́ỳ" * 6,                       # no codepoint before that takes them
    "growing": "क़ख़ग़ज़" * 8,                 # three bytes to six: past 28 bytes a chunk
    "growing far": "\U0001d15e\U0001d160" * 8,                 # four bytes to eight and twelve
    "long": "ậ́̀̄̆̇" * 4,  # more than fifteen bytes in one stretch
    "jamo": "한글" * 5,
    "mixed": "éक़q̣̇ ÅÅ1̖́" * 4,
}


@pytest.mark.parametrize("name", sorted(STRETCHES))
@pytest.mark.parametrize("edge", (0, 16, TILE, 2 * TILE))
def test_kept_stretches(built, name, edge):
    for shift in range(0, 17):
        text = "x" * max(0, edge - 8 + shift) + STRETCHES[name] + " tail"
        got = oracle_lib.device_nfc(text.encode(), reverse=bool(shift & 1))
        assert got == unicodedata.normalize("NFC", text).encode(), (shift, text[-60:])
