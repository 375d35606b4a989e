"""How the network's loader warp hands shared memory to the tensor cores (CPU: read from the
kernel's source and replayed).

Copies issued by the lanes (cp.async, st.shared) write through the generic proxy, the MMAs
read through the async proxy. A barrier alone does not order the two: each lane has to see
its copies land, fence the proxies, and only then arrive."""
from __future__ import annotations

import os
import random
import re

import pytest

from conftest import ROOT

CONV = os.path.join(ROOT, "discodj.jl_b200", "csrc", "conv_tc.cuh")


def _source():
    return re.sub(r"//[^\n]*", "", open(CONV).read())


def _constant(name):
    src = _source()
    v = re.search(rf"constexpr int {name} = (\w+);", src).group(1)
    return int(v if v.isdigit() else re.search(rf"#define {v} (\d+)", src).group(1))


def test_copied_planes_are_fenced_before_their_barrier_arrives():
    src = _source()
    # no arrival made by the copy unit itself: nothing could stand between copy and arrival
    assert "cp.async.mbarrier.arrive" not in src
    body = re.search(r"struct HandOver \{.*?\n\};", src, re.S).group(0)
    for method in ("push", "drain"):
        text = re.search(rf"void {method}\(.*?\n    \}}", body, re.S).group(0)
        at = [text.index(s) for s in ("cp_async_wait<", "fence_proxy_async_smem()", "mbar_arrive(")]
        assert at == sorted(at), method
    # every branch that copies by lane ends in a push
    for m in re.finditer(r"if \([^\n]*\) cp_async16\(|\n\s+cp_async16\(", src):
        assert "held.push(" in src[m.end():m.end() + 700]


def _replay(loader, mma, progress):
    """Runs the two roles in turn; False when neither can move."""
    running, still = [loader, mma], 0
    while running:
        before = progress()
        for g in list(running):
            if next(g, None) is None:
                running.remove(g)
        still = still + 1 if running and progress() == before else 0
        if still > 3:
            return False
    return True


def _forward(items, ring, behind):
    """items: (tiles, interior) per column segment, as k_conv3_tc walks them."""
    full, freed = set(), [0]

    def loader():
        held, k = [], 0
        for tiles, interior in items:
            if interior:
                full.update(held)
                held = []
            for _ in range(tiles + 2):
                while k - ring >= freed[0]:
                    yield 1
                if interior:
                    full.add(k)
                else:
                    held.append(k)
                    if len(held) > behind:
                        full.add(held.pop(0))
                k += 1
        full.update(held)

    def mma():
        base = 0
        for tiles, _ in items:
            while base not in full:
                yield 1
            for u in range(-1, tiles + 1):   # plane u is at base + u + 1; the next is waited for first
                while u < tiles and base + u + 2 not in full:
                    yield 1
                freed[0] = base + u + 2
            base += tiles + 2

    return _replay(loader(), mma(), lambda: (len(full), freed[0]))


def _gradient(items, tma, ring, buffers, behind):
    """The weight gradient's loader and MMA role (k_conv3_wgrad)."""
    x, y, freed_x, freed_y = set(), set(), set(), [0]

    def loader():
        held, kx, ky = [], 0, 0

        def push(where, what):
            held.append((where, what))
            if len(held) > behind:
                w, v = held.pop(0)
                w.add(v)

        def drain():
            for w, v in held:
                w.add(v)
            held.clear()

        for tiles, interior in items:
            interior = interior and tma
            if interior:
                drain()
            for i in range(tiles):
                for _ in range(3 if i == 0 else 1):
                    while kx >= ring and kx - ring not in freed_x:
                        yield 1
                    x.add(kx) if interior else push(x, kx)
                    kx += 1
                while ky - buffers >= freed_y[0]:
                    yield 1
                y.add(ky) if tma else push(y, ky)
                ky += 1
        drain()

    def mma():
        base, ky = 0, 0
        for tiles, _ in items:
            while ky not in y or any(base + j not in x for j in range(3)):
                yield 1
            for i in range(tiles):
                while i + 1 < tiles and (ky + 1 not in y or base + i + 3 not in x):
                    yield 1
                freed_x.add(base + i)
                ky += 1
                freed_y[0] = ky
            freed_x.update((base + tiles, base + tiles + 1))
            base += tiles + 2

    return _replay(loader(), mma(), lambda: (len(x), len(y), len(freed_x), freed_y[0]))


@pytest.mark.parametrize("seed", range(4))
def test_held_back_planes_never_stall_the_ring(seed):
    """The loader may block on a slot while it still holds planes back: the MMAs that free the
    slot must not need one of those. One more plane held back than the ring allows does stall."""
    rng = random.Random(seed)
    ring, behind = _constant("kRing"), _constant("kBehind")
    wring, wy, wbehind = _constant("kWRing"), _constant("kWY"), _constant("kWBehind")
    cases = [[(rng.choice([1, 2, 3, 4, 5, 15, 16]), rng.random() < 0.5) for _ in range(rng.randint(1, 7))]
             for _ in range(300)]
    assert all(_forward(c, ring, behind) for c in cases)
    assert all(_gradient(c, tma, wring, wy, wbehind) for c in cases for tma in (False, True))
    assert not all(_forward(c, ring, ring - 1) for c in cases)
    assert not all(_gradient(c, tma, wring, wy, 4) for c in cases for tma in (False, True))
