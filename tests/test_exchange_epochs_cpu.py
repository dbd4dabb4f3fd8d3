"""The numbers of the whole-device exchange (``GridX`` in
``csrc/pcg_exchange.cuh``), modelled and checked exhaustively on the CPU.

A word holds its payload and the number of its exchange; a reader takes it when
the number is the one it expects.  A launch starts from the number the launch
before left.  The model runs two CTAs through two launches of ``B`` exchanges over
every interleaving of their steps (reading the start number, writing a word,
taking or giving up a wait), a CTA that starts after the other gave up included,
and checks that no CTA takes a word of an earlier launch.

``clear``: after a launch in which a wait gave up the host clears the words and
the number (``collect``).  Otherwise CTA 0 publishes a number further on when it
gives up; a CTA that starts after that writes words of the very numbers that the
next launch uses, which the model finds.
"""
from collections import deque

import pytest

START, WRITE, WAIT, DONE, GAVE_UP = range(5)


def stale_reads(B, clear, give_up):
    """(states where a CTA takes an earlier launch's word, number of states)"""
    skip = 2 * B + 16
    # launch, the CTAs' (mode, exchange, number), words by parity and CTA as (number, launch), the number left
    start = (0, ((START, 0, 0),) * 2, (((0, -1),) * 2,) * 2, 0)
    seen, q, bad = {start}, deque([start]), []
    while q:
        st = q.popleft()
        launch, cta, words, left = st
        nxt = []
        if all(m in (DONE, GAVE_UP) for m, _, _ in cta):
            if launch == 0:
                if clear and any(m == GAVE_UP for m, _, _ in cta):
                    nxt.append((1, ((START, 0, 0),) * 2, (((0, -1),) * 2,) * 2, 0))
                else:
                    nxt.append((1, ((START, 0, 0),) * 2, words, left))
        else:
            for i in (0, 1):
                mode, e, ep = cta[i]

                def go(new, w=words, n=left):
                    nxt.append((launch, tuple(new if k == i else cta[k] for k in (0, 1)), w, n))

                if mode == START:
                    go((WRITE, 0, left + 1))
                elif mode == WRITE:
                    par = ep & 1
                    row = tuple((ep, launch) if k == i else words[par][k] for k in (0, 1))
                    go((WAIT, e, ep), w=tuple(row if p == par else words[p] for p in (0, 1)))
                elif mode == WAIT:
                    number, by = words[ep & 1][1 - i]
                    if number == ep:
                        if by != launch:
                            bad.append(st)
                        last = e + 1 == B
                        go((DONE if last else WRITE, e + 1, ep + 1), n=ep + 1 if last and i == 0 else left)
                    if give_up and launch == 0:
                        go((GAVE_UP, e, ep), n=left if clear or i else ep + skip)
        for s in nxt:
            if s not in seen:
                seen.add(s)
                q.append(s)
    return bad, len(seen)


@pytest.mark.parametrize("B", [1, 2, 3])
def test_no_word_of_an_earlier_launch_is_taken(B):
    for give_up in (False, True):
        bad, n = stale_reads(B, clear=True, give_up=give_up)
        assert not bad, bad[:2]
        assert n > 10 * B


@pytest.mark.parametrize("B", [1, 2])
def test_the_model_sees_a_number_published_ahead(B):
    assert not stale_reads(B, clear=False, give_up=False)[0]
    assert stale_reads(B, clear=False, give_up=True)[0]
