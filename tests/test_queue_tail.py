"""The chunk queue's tail word (swr_queue.h): on the host, its two fields under as many claims in flight as the kernels
can make, at the largest capacity and at the chunk limit; on the GPU, a draw of more large triangles than the
slot field counts."""
import os
import subprocess

import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import CLIP_FROM_OBJECT, GpuRenderer, assert_visbuffer_equal, render_oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <vector>
#include "glimpsw_gb300/csrc/swr_queue.h"
using namespace swr;

struct Claim { unsigned long long word; uint32_t slots; };

// `triangles` claims of `slots` slots and up to maxChunks chunks against a queue of `capacity`, each claim without room
// taken back only after `delay` later claims. Returns the tail, having checked every slot handed out.
static unsigned long long run(uint32_t capacity, uint32_t slots, uint32_t maxChunks, unsigned long long triangles, size_t delay,
                              unsigned long long start) {
    unsigned long long tail = start, expect = start;
    bool full = false;
    std::deque<unsigned long long> back;
    uint32_t seed = 1;
    for (unsigned long long i = 0; i < triangles; i++) {
        seed = seed * 1664525u + 1013904223u;
        const uint32_t chunks = 1 + (seed >> 8) % maxChunks;
        const unsigned long long claim = queue_claim(slots, chunks), old = tail;
        tail += claim;
        assert(queue_slots(tail) == queue_slots(old) + slots && queue_chunks(tail) == queue_chunks(old) + chunks);  // no carry
        if (queue_fits(queue_slots(old), queue_chunks(old), slots, capacity)) {
            assert(!full && old == expect);  // nothing fits after a claim that did not, and its slots are the next
            assert(queue_slots(old) + slots <= capacity);
            expect = tail;
        } else {
            full = true;
            back.push_back(claim);
        }
        if (back.size() > delay) tail -= back.front(), back.pop_front();
    }
    for (unsigned long long c : back) tail -= c;
    assert(tail == expect && queue_slots(tail) <= capacity);
    return tail;
}

int main() {
    const size_t inFlight = kQueueWarps * 32;
    for (uint32_t slots = 1; slots <= 2; slots++) {
        for (uint32_t capacity : { 1u, 2u, 13u, 1000u, kQueueMaxCapacity - 1, kQueueMaxCapacity })  // far past 2^24 claims
            assert(queue_slots(run(capacity, slots, 100, capacity > 1000 ? 40000000ull : 20000ull, inFlight - 1, 0)) == capacity / slots * slots);
        // close to the chunk limit, every triangle as many chunks as one can have
        run(kQueueMaxCapacity, slots, 1u << 17, 3000000, inFlight - 1, queue_claim(1000, 0) | (kQueueChunkLimit - 5000000));
    }
    puts("ok");
}
"""


def test_fields_do_not_carry(tmp_path):
    src, exe = tmp_path / "queue.cpp", tmp_path / "queue"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", ROOT, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


@pytest.mark.gpu
def test_more_large_triangles_than_slots():
    """131,080 meshlets of 128 triangles above 16 tiles, all but the first behind it: 2^24 + 1,024 triangles for a queue
    of a fixed 13, then of a quarter of them, then (it overflowed) of its largest capacity."""
    m = np.zeros(131_080, dtype=scenes.MESHLET_DTYPE)
    side = 8
    g = np.linspace(-0.95, 0.95, side, dtype=np.float32)
    x, y = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    cell = np.arange(side * side).reshape(side, side)
    a, b, c, d = cell[:-1, :-1].ravel(), cell[1:, :-1].ravel(), cell[:-1, 1:].ravel(), cell[1:, 1:].ravel()
    tri = np.concatenate([np.stack([a, b, c], 1), np.stack([b, d, c], 1)])
    tri = np.concatenate([tri, tri[: 128 - len(tri)]])
    w = np.where(np.arange(len(m)) == 0, 1.0, 2.0).astype(np.float32)[:, None]  # powers of two: the same projection
    m["Positions"][:, 0], m["Positions"][:, 1], m["Positions"][:, 2] = x * w, y * w, w
    m["NumVertices"], m["NumTriangles"], m["AlphaCutoff"] = 64, 128, 255
    m["Indices"] = tri.T.astype(np.uint8)
    mats = np.zeros(1, dtype=scenes.MATERIAL_DTYPE)
    mats["alpha_cutoff"], mats["is_double_sided"] = 255, 1
    assert len(m) * 128 > 1 << 24
    size = 184  # cells of 25 pixels: boxes of 7 x 7 tiles
    ofb, oc = render_oracle(m[:1], mats, CLIP_FROM_OBJECT, size, size)
    assert oc[1] == 128
    r = GpuRenderer(m, mats)
    for capacity in (13, 0, 0):
        r.rast.set_queue_capacity(capacity)
        fb, counters = r.render(CLIP_FROM_OBJECT, size, size)
        assert_visbuffer_equal(fb, ofb)
        assert list(counters[:3]) == [128 * len(m), 128 * len(m), 0]
