"""The tags of the one-launch PCG's reductions after a wait that ran out (skt_rules.hpp, compiled for the host):
the exchange played by a model of the blocks, one step of one block at a time in a random order, in which a
block may give up waiting whenever the partial it waits for has not come. After an abandoned launch the next
one must never take one of its partials for its own."""
import ctypes
import random
import subprocess

import pytest

from skewtcloudsim_gb300 import build


@pytest.fixture(scope="module")
def tag_after(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text('#include "skt_rules.hpp"\nextern "C" unsigned after(unsigned t, int s) { return skt::tag_after(t, s != 0); }\n')
    so = str(d / "rules.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", build.CSRC, str(d / "rules.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).after
    f.restype = ctypes.c_uint
    f.argtypes = [ctypes.c_uint, ctypes.c_int]
    return lambda t, s: f(t, int(s))


def launch(inbox, nb, first, reductions, rng, may_give_up, serial):
    """One launch; returns block 0's last tag, whether it gave up, and whether any block took a stale partial.
    inbox[parity][to][from] = (tag, launch that sent it)."""
    tag, sent, stuck, stale = [first] * nb, [False] * nb, [False] * nb, False
    late = rng.randrange(nb) if may_give_up else -1
    live = set(range(nb))
    while live:
        b = rng.choice(sorted(live))
        if b == late and rng.random() < 0.9:  # this one is slow: others may have given up before it sends
            continue
        t = tag[b]
        if not sent[b]:
            for to in range(nb):
                inbox[t & 1][to][b] = (t, serial)
            sent[b] = True
            continue
        got = inbox[t & 1][b]
        if all(g[0] == t for g in got):
            stale |= any(g[1] != serial for g in got)
            if t - first + 1 == reductions:
                live.remove(b)
            else:
                tag[b], sent[b] = t + 1, False
        elif may_give_up and rng.random() < 0.1:
            stuck[b] = True
            live.remove(b)
    return tag[0], stuck[0], stale


def play(rule, seed):
    rng = random.Random(seed)
    nb = rng.randrange(2, 6)
    inbox = [[[(0, -1)] * nb for _ in range(nb)] for _ in range(2)]
    tag, abandoned = 0, False
    for serial in range(4):
        last, stuck, stale = launch(inbox, nb, tag + 1, rng.randrange(2, 6), rng, serial < 3, serial)
        if stale:
            return True, abandoned
        abandoned |= stuck
        tag = rule(last, stuck)
    return False, abandoned


def test_no_partial_of_an_abandoned_launch_is_taken(tag_after):
    results = [play(tag_after, seed) for seed in range(3000)]
    assert not any(stale for stale, _ in results)
    assert sum(a for _, a in results) > 500  # launches were abandoned
    # the model finds the fault where the tag is kept as block 0 left it
    assert any(play(lambda t, s: t, seed)[0] for seed in range(3000))
