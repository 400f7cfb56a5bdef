"""Calls that programs make on this framework, for timing them.

A case is one call of `gpu_bpe_tokenizer.Tokenizer` on text (or ids) in host memory: `encode_numpy`,
`encode_to_device`, `encode_batch`, `encode_batch_to_device` or `decode_bytes`.  Between them the cases
take the five vocabulary families, single texts from a chat line to a 32 MiB corpus file, batches from a
handful of prompts to thousands of documents, `str` as well as `bytes`, results on the host and on the
GPU, and both directions.  Vocabularies and texts are those of `graphtok_b200.synth` (the Gemma-3-shaped
vocabulary, which has no synthetic training there, is the committed one of the tests).

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs and tokenizer, as a program has them in hand before the call
    run(state)          the call
    work(case)          bytes that the call cannot do without
    tolerance(case)     ids and bytes are exact
"""
import functools
import math
import os
import unicodedata

import numpy as np

import graphtok_b200
from graphtok_b200 import synth
from graphtok_b200.gpu_bpe_tokenizer import Tokenizer

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(graphtok_b200.__file__)))

#: vocabulary of each family
VOCAB = {"gpt2": "cfg0", "llama3": "cfg1", "qwen25": "cfg3", "deepseek": "cfg5"}
#: text kind -> (text configuration of the generator, bytes of it that are kept to cut inputs from).  None of it is a text
#: that a vocabulary was trained on.
KINDS = {"english": (0, 16 << 20), "multilingual": (1, 16 << 20), "code_cjk": (3, 16 << 20), "mixed_runs": (4, 48 << 20)}
#: kinds of text each family is given in draw()
USUAL = {"gpt2": ("english",), "llama3": ("multilingual", "mixed_runs", "english"), "qwen25": ("code_cjk", "english"),
         "deepseek": ("multilingual", "code_cjk"), "gemma": ("multilingual", "english")}
CORPUS_SEED = 21
PIECE = 1 << 18          # a text longer than this is put together from pieces of this length
#: bytes of text behind one id, as measured, and the first guess at the text that gives a number of ids
ID_BYTES = {("llama3", "multilingual"): 5.1, ("llama3", "mixed_runs"): 2.4, ("deepseek", "multilingual"): 4.9, ("deepseek", "code_cjk"): 3.2,
            ("gemma", "multilingual"): 2.7, ("gemma", "english"): 2.6}


def listed():
    return [
        # One line of a chat: the shortest text that is ever sent by itself, where launch and wait are the whole time.
        {"name": "chat_line", "op": "encode", "family": "llama3", "kind": "english", "ids": 14, "as_str": True},
        # A chat message of a paragraph or two (about 1 KB), in a script other than Latin as often as not.
        {"name": "chat_message", "op": "encode", "family": "deepseek", "kind": "multilingual", "ids": 211, "as_str": True},
        # A prompt with a source file in it (16 KB); the vocabulary normalises (NFC), so the text passes the normalisation kernels.
        {"name": "code_prompt", "op": "encode", "family": "qwen25", "kind": "code_cjk", "ids": 3889, "as_str": True},
        # The longest prompt that is served: pasted logs, base64 blocks, long runs of one character; about 310 KB.
        {"name": "long_prompt", "op": "encode", "family": "llama3", "kind": "mixed_runs", "ids": 128001, "as_str": False},
        # A document of the headline benchmark's size: multilingual, 4.5 MB, ids to host memory.
        {"name": "document", "op": "encode", "family": "llama3", "kind": "multilingual", "ids": 892973, "as_str": False},
        # A repository dump of 8 MiB for the model on the same GPU: decomposed characters in it, ids stay on the device.
        {"name": "code_to_device", "op": "encode_to_device", "family": "qwen25", "kind": "code_cjk", "ids": 1972001, "as_str": False},
        # A chapter (300 KB) for a model with a character-level vocabulary (spaces as U+2581, byte fallback).
        {"name": "chapter_gemma", "op": "encode", "family": "gemma", "kind": "multilingual", "ids": 111007, "as_str": True},
        # A corpus file of 32 MB, the largest single call: everything that is awkward in real text mixed in one stream.
        {"name": "corpus_file", "op": "encode", "family": "llama3", "kind": "mixed_runs", "ids": 14000003, "as_str": False},
        # A shard of a pre-training set: thousands of documents (27 MB) as a list of Python strings, one call.
        {"name": "training_shard", "op": "encode_batch", "family": "gpt2", "kind": "english", "docs": 8192, "ids": 6150011, "as_str": True},
        # What a serving scheduler collects between two steps: some dozens of requests, ids wanted on the device.
        {"name": "request_batch", "op": "encode_batch_to_device", "family": "deepseek", "kind": "multilingual", "docs": 48, "ids": 32749, "as_str": True},
        # One finished reply, a list of some 300 ids from a sampler, to text.
        {"name": "reply_decode", "op": "decode", "family": "llama3", "kind": "english", "bytes": 1361, "as_list": True},
        # A tokenised document back to text.
        {"name": "document_decode", "op": "decode", "family": "llama3", "kind": "multilingual", "bytes": 4500001, "as_list": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("encode", "encode", "encode", "encode_to_device", "encode_batch", "encode_batch_to_device", "decode"))
    family = rng.choice(tuple(USUAL))
    case = {"op": op, "family": family, "kind": rng.choice(USUAL[family])}
    if op == "decode":
        case["bytes"] = _log(rng, 40, 6 << 20)
        case["as_list"] = case["bytes"] < 16384
    elif op.startswith("encode_batch"):
        case["docs"] = _log(rng, 2, 4096)
        case["ids"] = case["docs"] * _log(rng, 30, 1200) + rng.randrange(17)
        case["as_str"] = rng.random() < 0.5
    else:
        case["ids"] = _log(rng, 5, 2800000)
        case["as_str"] = case["ids"] < 16384 or rng.random() < 0.25
    return case


@functools.lru_cache(maxsize=None)
def _tokenizer(family):
    # one per vocabulary and GPU, kept for the life of the program, as a server keeps it
    path = os.path.join(ROOT, "tests", "golden", "tiny_gemma.json") if family == "gemma" else synth.vocab_path(VOCAB[family])
    return Tokenizer(path, max_input_chars=1 << 20)


@functools.lru_cache(maxsize=None)
def _corpus(kind):
    config, size = KINDS[kind]
    return synth.text(config, CORPUS_SEED, size)


def _cut(corpus, at, n):
    """About n bytes from `at` on, whole UTF-8 characters."""
    end = at + n
    while at < end and corpus[at] & 0xC0 == 0x80:
        at += 1
    while end < len(corpus) and end > at and corpus[end] & 0xC0 == 0x80:
        end -= 1
    return corpus[at:end]


def _text(kind, n, rng):
    corpus = _corpus(kind)
    return b"".join(_cut(corpus, int(rng.integers(0, len(corpus) - min(PIECE, n - i))), min(PIECE, n - i)) for i in range(0, n, PIECE))


def _prefix(count, text, want):
    """A prefix of `text` that gives exactly `want` ids, whole characters; None where the search ends without one."""
    lo, hi, n_lo, n_hi = 0, len(text), 0, count(text)
    if n_hi <= want:
        return text if n_hi == want else None
    for step in range(200):
        # interpolation and bisection in turn: ids follow the length closely, but for runs of one character
        share = (want - n_lo) / (n_hi - n_lo) if step % 3 < 2 and n_hi > n_lo else 0.5
        mid = lo + min(max(int((hi - lo) * share), 1), hi - lo - 1) if hi - lo > 1 else hi
        while mid < hi and text[mid] & 0xC0 == 0x80:
            mid += 1
        if mid >= hi:                       # at most one character is left between lo and hi
            mid = hi - 1
            while mid > lo and text[mid] & 0xC0 == 0x80:
                mid -= 1
            if mid <= lo:
                return None
        n = count(text[:mid])
        if n == want:
            return text[:mid]
        if n < want:
            lo, n_lo = mid, n
        else:
            hi, n_hi = mid, n
    return None


def _text_of(tok, family, kind, ids, rng):
    """A text of exactly `ids` ids, so that every seed's result has the same shape."""
    room = 1.08 * ID_BYTES.get((family, kind), 4.4)
    while True:
        text = _prefix(lambda t: tok.encode_numpy(t).size, _text(kind, int(room * ids) + 64, rng), ids)
        if text is not None:
            return text
        room *= 1.1


def _documents(tok, family, kind, docs, ids, rng):
    """`docs` documents of `ids` ids in all.  Lengths as in the batch configuration: log-normal, spread over two orders of magnitude."""
    share = np.clip(rng.lognormal(0.0, 1.0, docs), 0.03, 16.0)
    corpus = _corpus(kind)
    at = rng.integers(0, len(corpus) - (1 << 20), docs)
    size = ID_BYTES.get((family, kind), 4.4) * (ids - 1.0 * ids / docs) / share[:-1].sum()     # bytes of a document of share 1
    while True:
        got = [_cut(corpus, int(a), max(1, int(size * s))) for a, s in zip(at[:-1], share[:-1])]
        left = ids - tok.encode_batch(got)[0].size
        if 0 < left < 3.0 * ids / docs + 64:
            return got + [_text_of(tok, family, kind, left, rng)]
        size *= max(0.5, min(2.0, (ids - 1.0 * ids / docs) / max(1, ids - left)))


def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    tok = _tokenizer(case["family"])
    state = {"call": getattr(tok, {"encode": "encode_numpy", "decode": "decode_bytes"}.get(case["op"], case["op"])), "op": case["op"]}
    if case["op"] == "decode":
        text = _text(case["kind"], case["bytes"], rng).ljust(case["bytes"])     # whole characters, blanks up to the exact length
        if case["family"] == "qwen25":
            text = unicodedata.normalize("NFC", text.decode("utf-8")).encode("utf-8").ljust(case["bytes"])
        ids = tok.encode_numpy(text)
        state["input"] = ids.tolist() if case["as_list"] else ids
    elif "docs" in case:
        docs = _documents(tok, case["family"], case["kind"], case["docs"], case["ids"], rng)
        state["input"] = [d.decode("utf-8") for d in docs] if case["as_str"] else docs
    else:
        text = _text_of(tok, case["family"], case["kind"], case["ids"], rng)
        state["input"] = text.decode("utf-8") if case["as_str"] else text
    return state


def run(state):
    result = state["call"](state["input"])
    return np.frombuffer(result, dtype=np.uint8) if state["op"] == "decode" else result


def work(case):
    """Text read once, ids written once (or the other way round), four bytes an id; document offsets in and out."""
    each = ID_BYTES.get((case["family"], case["kind"]), 4.4)
    if case["op"] == "decode":
        return {"bytes": case["bytes"] * (1.0 + 4.0 / each), "flops": 0.0}
    return {"bytes": case["ids"] * (each + 4.0) + 8.0 * (case.get("docs", -1) + 1), "flops": 0.0}


def tolerance(case):
    return "exact"
