"""CPU: the tagged vectors of the decode kernel have a single buffer each, so whoever publishes a word has to know that the word before it, in the same place,
was read by everybody who polls for it: a reader that comes later never sees its tag again and gives up. This follows what every CTA of a launch
publishes and what it waited for by then, for every shape that a kernel is built for."""
import os
import re

import numpy as np
import pytest

import geometry

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flint_b200", "csrc")


class Launch:
    """Vector clocks of the CTAs: clock[a][b] is the last event of CTA b that is known to lie before whatever CTA a does next."""

    def __init__(self, sms):
        self.clock = np.zeros((sms, sms), dtype=np.int64)
        self.words = {}       # (buffer, word group) -> [publisher's clock at that time, [(reader, its event)]]
        self.late = []        # (buffer, word group, publisher, reader that it knew nothing of)

    def publish(self, cta, key):
        """`cta` writes a group of words of its own"""
        for reader, event in self.words.get(key, (None, ()))[1]:
            if reader != cta and self.clock[cta, reader] < event:
                self.late.append((*key, cta, reader))
        self.clock[cta, cta] += 1
        self.words[key] = [self.clock[cta].copy(), []]

    def read(self, cta, keys):
        """`cta` waits for the present words"""
        if keys:
            self.clock[cta] = np.maximum(self.clock[cta], np.max([self.words[k][0] for k in keys], axis=0))
            self.clock[cta, cta] += 1
            for k in keys:
                self.words[k][1].append((cta, int(self.clock[cta, cta])))


def _rank(shape):
    """(query heads, kv heads, ranks) of the ranks that a shape's kernel serves"""
    kd, ko, _, hd, r = shape
    for nh in range(r, ko // hd + 1, r):
        if kd % (nh * hd) == 0 and {geometry.o_window(nh * hd, i)[0] for i in range(kd // (nh * hd))} == {ko}:
            return nh, nh // r, kd // (nh * hd)
    raise AssertionError(shape)


def _follow(shape, sms, chunks, layers=3, zeros_published=False):
    """A token as the kernel's consumers go through it. zeros_published: CTA 0 publishes zeros for the columns of the O window that are not this rank's, ahead of its
    attention, and the O phase waits for them: what the kernel must not do."""
    kd, ko, kf, hd, r = shape
    nh, nkv, _ = _rank(shape)
    unit = max(geometry.tile_rt(ko), geometry.tile_rt(kf))
    qkv = geometry.cta_rows((nh + 2 * nkv) * hd, geometry.tile_rt(kd), sms)
    own = geometry.cta_rows(kd, unit, sms)
    gu = geometry.cta_rows(2 * kf, geometry.tile_rt(kd), sms)
    owners = {n: [b for b in range(sms) if at[b][1] > at[b][0]] for n, at in (("qkv", qkv), ("own", own), ("gu", gu))}

    def rows_of(first, heads):                 # who publishes a word of these heads of the QKV rows
        return [b for b in owners["qkv"] if qkv[b][0] < (first + heads) * hd and qkv[b][1] > first * hd]
    queries = [rows_of(g * r, r) for g in range(nkv)]
    new = [rows_of(nh + g, 1) + rows_of(nh + nkv + g, 1) for g in range(nkv)]       # this step's key and value: the chunk with its position reads them
    items = [(i % sms, i // chunks, i % chunks) for i in range(nkv * chunks)]      # CTA, kv head, chunk
    padded = zeros_published and geometry.o_window(nh * hd, 0)[0] > nh * hd
    run = Launch(sms)
    for layer in range(layers):
        for b in owners["qkv"]:
            if layer:
                run.read(b, [("h", o) for o in owners["own"]])
            run.publish(b, ("q", b))
        if padded:
            run.publish(0, ("ao", "zeros"))
        for b, g, c in items:
            run.read(b, [("q", o) for o in queries[g] + (new[g] if c == chunks - 1 else [])])
            if chunks > 1:
                run.publish(b, ("part", (g, c)))
        for b, g, c in items:
            if chunks > 1:
                run.read(b, [("part", (g, i)) for i in range(chunks)])
            run.publish(b, ("ao", (g, c)))
        for b in owners["own"]:
            run.read(b, [("ao", (g, c)) for _, g, c in items] + ([("ao", "zeros")] if padded else []))
            run.publish(b, ("h", b))
        for b in owners["gu"]:
            run.read(b, [("h", o) for o in owners["own"]])
            run.publish(b, ("act", b))
        for b in owners["own"]:
            run.read(b, [("act", o) for o in owners["gu"]])
            run.publish(b, ("h", b))
    return run.late


@pytest.mark.parametrize("sms", [132, 148, 160])
@pytest.mark.parametrize("shape", geometry.decode_shapes(), ids=str)
def test_nobody_publishes_over_a_word_that_is_still_polled_for(shape, sms):
    for chunks in {1, max(1, min(64, sms // _rank(shape)[1]))}:
        assert _follow(shape, sms, chunks) == []


def test_zeros_published_by_a_cta_that_has_not_waited_are_found():
    """The two-rank slice of the small decoder with heads of 80, where CTA 0 of 148 has no rows: it would publish the next layer's zeros straight behind its own
    attention of this one. (Where CTA 0 has rows, as in the 3B-class shape over 8, waiting for their input holds it back.)"""
    late = _follow((640, 384, 512, 80, 4), 148, 4, zeros_published=True)
    assert late and all(w[:3] == ("ao", "zeros", 0) for w in late)
    assert _follow((2560, 384, 1024, 80, 4), 148, 4, zeros_published=True) == []


def test_attention_output_is_published_by_the_attention_alone():
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "fb_decode.cuh")).read())
    stores = re.findall(r"ll_store2?\(\s*(\w+\.ao_ll)", code)
    assert stores and set(stores) == {"a.ao_ll"}          # AttnArgs, in attention_phase


@pytest.mark.parametrize("shape", geometry.decode_shapes(), ids=str)
def test_o_phase_waits_for_exactly_the_words_of_the_own_heads(shape):
    kd, ko, _, hd, _ = shape
    nh, _, ranks = _rank(shape)
    for rank in range(ranks):
        cols, off, first, end = geometry.o_window(nh * hd, rank)
        assert cols == ko and 0 <= off and off + nh * hd <= ko
        assert (4 * first, 4 * end) == (off, off + nh * hd)          # four columns a pair of words
    assert ranks > 1 or (first, end) == (0, ko // 4)
