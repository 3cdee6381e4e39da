"""The protocol of the wide sweeps' rings (csrc/wcns_ring.h), checked on the host
against the order that the kernel's barriers give: an entry counts as read only
when its read happens before the publication whichever warp is late, the writer
waits for exactly what it overwrites, and a chain of CTAs always gets to its end.

Order of the reader's CTA (k_sweep_wide.cu): the compute warps join the barrier of
every plane in turn; ring warp T & 1 joins those of its own parity and fetches plane
T between the barriers of T - 2 and T; a publication follows its own warp's fetch."""
import subprocess

import pytest

from wcns_b200.build import CSRC

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <vector>
#include "wcns_ring.h"
using namespace wcns;

// fetch(a) happens before the end of fetch(b): the same warp's earlier one, or by way
// of barrier a, which fetch(a) precedes, and barrier b - 2, which precedes fetch(b)
static bool before(int a, int b) { return (a & 1) == (b & 1) ? a <= b : a <= b - 2; }

static int published(int sdel, int np) {
    for (int sf = 0; sf < np; sf++)
        if (ring_publishes(sf))
            for (int e = 0; e < ring_read(sf); e++)
                if (!before(e + 1 + sdel, sf + 1 + sdel)) {
                    printf("entry %d may be unread when %d are published after entry %d\n", e, ring_read(sf), sf);
                    return 1;
                }
    return 0;
}

static int overwritten(int ringn, int np) {
    for (int sf = 0; sf < np; sf += RING_CHECK)
        for (int x = 0; x < RING_CHECK; x++)
            if (sf + x >= ringn && sf + x - ringn >= ring_room(sf, ringn)) {
                printf("entry %d is overwritten with %d read\n", sf + x - ringn, ring_room(sf, ringn));
                return 1;
            }
    return 0;
}

// G chunks over Gc CTAs, each later segment of a CTA `delay` planes behind: rounds in
// which every CTA goes as far as it can alone (order: up or down) until all are done.
// step: barriers passed.  Plane T of a CTA needs the neighbour's entry of plane T - 1,
// written in its step T - 1; entries are written in the step of their plane.
static int runs_to_the_end(int G, int Gc, int np, int ringn, int delay, bool up, bool forward) {
    const int nsegmax = (G + Gc - 1) / Gc, ns = np + (nsegmax - 1) * delay;
    auto sdel = [&](int q) { return (forward ? q / Gc : nsegmax - 1 - q / Gc) * delay; };
    std::vector<int> step(Gc, 0), wrote(G, 0), pub(G, 0);  // entries written to the next chunk, and published by it
    auto next = [&](int q) { return forward ? q + 1 : q - 1; };
    auto prev = [&](int q) { return forward ? q - 1 : q + 1; };
    auto inside = [&](int q) { return q >= 0 && q < G; };
    auto advance = [&](int c) {
        const int s = step[c];  // the barrier to pass: plane s's terms must be in
        if (s >= ns) return false;
        for (int q = c; q < G; q += Gc) {
            const int in = s - 1 - sdel(q);  // entry of plane s
            if (inside(prev(q)) && in >= 0 && in < np && wrote[prev(q)] <= in) return false;
            const int sf = s - sdel(q);
            if (inside(next(q)) && sf % RING_CHECK == 0 && sf >= 0 && sf < np && ring_room(sf, ringn) > 0 && pub[q] < ring_room(sf, ringn)) return false;
        }
        for (int q = c; q < G; q += Gc) {
            const int in = s - 1 - sdel(q), sf = s - sdel(q);
            if (inside(prev(q)) && in >= 0 && in < np && ring_publishes(in)) pub[prev(q)] = ring_read(in);
            if (sf >= 0 && sf < np) wrote[q] = sf + 1;
        }
        step[c]++;
        return true;
    };
    for (;;) {
        bool moved = false, done = true;
        for (int x = 0; x < Gc; x++) {
            const int c = up ? x : Gc - 1 - x;
            while (advance(c)) moved = true;
            done = done && step[c] >= ns;
        }
        if (done) return 0;
        if (!moved) {
            printf("%d chunks on %d CTAs, %d planes, ring %d, delay %d: stuck\n", G, Gc, np, ringn, delay);
            return 1;
        }
    }
}

int main() {
    int bad = 0;
    for (int np : {1, 7, 8, 9, 33, 64, 200})
        for (int sdel : {0, 8, 24}) bad |= published(sdel, np);
    for (int ringn : {32, 64, 128}) bad |= overwritten(ringn, 500);
    for (int np : {5, 31, 32, 40, 41, 113, 200})
        for (int delay : {0, 8, 40, 96})
            for (int G : {2, 3, 8, 17})
                for (int fold : {1, 2, 3, 8})
                    for (int o = 0; o < 4; o++) {
                        int ringn = 32;
                        while (ringn < delay + 32) ringn *= 2;
                        bad |= runs_to_the_end(G, (G + fold - 1) / fold, np, ringn, fold > 1 ? delay : 0, o & 1, o & 2);
                    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("rings")
    (d / "rings.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "rings.cpp"), "-o", str(d / "rings")], check=True)
    return str(d / "rings")


def test_ring_protocol(model):
    r = subprocess.run([model], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:]
