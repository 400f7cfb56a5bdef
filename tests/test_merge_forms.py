"""The forms of the merge kernels' work, one thread per pre-token, a team of lanes per pre-token, and teams over the one list of all
lengths that the single-block kernel has, each with its threads in order and in reverse (a step that depends on their order is a
race on the GPU), against the oracle where they can go wrong: lengths at the edges of the classes and mixed, list sizes at the
edges of a call, and vocabularies whose ranks are not monotone."""
import itertools
import json
import random

import numpy as np
import pytest

import oracle_lib
from conftest import FAMILIES, tiny_vocab

LETTERS = "abcdefghijklmnopqrstuvwxyz"
CYRILLIC = "абвгдежзийклмнопрстуфхцчшщъыьэюя"


RUNS = list(itertools.product(oracle_lib.Emul.FORMS, (False, True)))


def word(rng, size, alphabet):
    """A word of `size` bytes as UTF-8 (one ASCII letter more where the characters do not fit exactly)."""
    w = "".join(rng.choice(alphabet) for _ in range(size // len(alphabet[0].encode())))
    return w + "q" * (size - len(w.encode()))


@pytest.mark.parametrize("family", FAMILIES)
@pytest.mark.parametrize("alphabet", (LETTERS, "eta", CYRILLIC))
def test_lengths_at_the_edges_of_the_classes(emuls, oracles, family, alphabet):
    rng = random.Random(11)
    e, o = emuls[family], oracles[family]
    for size in (2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 47, 48, 49, 62, 63, 64, 65):
        text = " ".join(word(rng, size - 1, alphabet) for _ in range(40)).encode()
        want = o.encode_normalized(text)
        for form, reverse in RUNS:
            assert np.array_equal(e.encode(text, reverse=reverse, form=form), want), (size, form, reverse)


@pytest.mark.parametrize("size", (9, 25, 40, 60))
@pytest.mark.parametrize("count", (1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 129))
def test_list_sizes_at_the_edges_of_a_call(emuls, oracles, size, count):
    rng = random.Random(100 * size + count)
    for family in ("gpt2", "llama3"):
        text = (" " + " ".join(word(rng, size, LETTERS) for _ in range(count))).encode()
        want = oracles[family].encode_normalized(text)
        for form, reverse in RUNS:
            assert np.array_equal(emuls[family].encode(text, reverse=reverse, form=form), want), (family, form, reverse)


@pytest.mark.parametrize("family", FAMILIES)             # with and without ignore_merges
@pytest.mark.parametrize("longest", (16, 32, 64))
def test_lists_of_mixed_lengths(emuls, oracles, family, longest):
    """Vocabulary tokens of more than 15 bytes among words of every length up to the class's: more than one call of 256."""
    rng = random.Random(longest)
    known = [b for b in oracle_lib.token_spellings(tiny_vocab(family)).values() if 15 < len(b) <= longest] if family == "llama3" else []
    known = known or [b" the"]
    text = b"".join(rng.choice(known) if rng.random() < 0.1 else b" " + word(rng, rng.randint(2, longest - 1), LETTERS).encode() for _ in range(600))
    want = oracles[family].encode_normalized(text)
    for form, reverse in RUNS:
        assert np.array_equal(emuls[family].encode(text, reverse=reverse, form=form), want), (form, reverse)


@pytest.mark.parametrize("seed", range(4))
def test_ranks_that_are_not_monotone(built, tmp_path, seed):
    """Rules in a random order: a rule's parts may be made by rules that come after it, new pairs may be lower than the merge
    that made them."""
    rng = random.Random(seed)
    j = json.load(open(tiny_vocab("gpt2"), encoding="utf-8"))
    rng.shuffle(j["model"]["merges"])
    path = str(tmp_path / "shuffled.json")
    json.dump(j, open(path, "w", encoding="utf-8"), ensure_ascii=False)
    e, o = oracle_lib.Emul(path), oracle_lib.Oracle(path)
    for alphabet in (LETTERS, "etaoin", "th", "e", CYRILLIC):
        text = " ".join(word(rng, rng.randint(2, 64), alphabet) for _ in range(300)).encode()
        want = o.encode_normalized(text)
        for form, reverse in RUNS:
            assert np.array_equal(e.encode(text, reverse=reverse, form=form), want), (alphabet, form, reverse)
