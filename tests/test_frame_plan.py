"""The host arithmetic of a frame's and a replay's launch (csrc/rtb_plan.h, compiled here for the
host): over frame sizes from one pixel to beyond 4K and 1 to 512 samples, and whichever of the
buffers can be had, the path slots that the launch uses lie inside the buffer that was asked for
last, the queue's items cover every sample once, and a frame without slots takes the form that
needs none."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "master-rad_b200", "csrc")
SOURCE = r"""
#include "rtb_plan.h"
using namespace rtb;
struct Out { long long block, slots, grid, items, split, tail_pixels, tail_bytes, path_bytes, had_tail, had_paths; };
extern "C" void settle(int block, int sm_count, long long resident, long long pixels, int spp, long long tail,
                      long long tail_limit, long long path_limit, Out* o) {
  FrameShape f;
  f.block = block;
  f.sm_count = sm_count;
  f.spp = spp;
  f.pixels = pixels;
  f.resident = resident;
  f.set_tail(tail);
  *o = Out{};
  settle_frame(
      f, [&](size_t n) { return (long long)n <= tail_limit ? (o->had_tail = (long long)n, true) : false; },
      [&](size_t n) { return (long long)n <= path_limit ? (o->had_paths = (long long)n, true) : false; },
      [&] { return resident / 2; });
  o->block = f.block;
  o->slots = f.slots;
  o->grid = f.grid;
  o->items = f.items;
  o->split = f.split;
  o->tail_pixels = f.tail_pixels;
  o->tail_bytes = (long long)f.tail_bytes();
  o->path_bytes = f.block == kBlock ? (long long)(f.grid * block_path_bytes(f.slots)) : 0;
}
extern "C" void replay(long long samples, int max_depth, int sm_count, long long* o) {
  const ReplayShape r(samples, max_depth, sm_count);
  o[0] = r.grid;
  o[1] = r.slots;
  o[2] = (long long)r.path_bytes;
  o[3] = (long long)r.vertex_bytes;
  o[4] = (long long)(r.grid * block_path_bytes(r.slots));
}
"""
FIELDS = ("block", "slots", "grid", "items", "split", "tail_pixels", "tail_bytes", "path_bytes", "had_tail",
          "had_paths")


class Out(C.Structure):
    _fields_ = [(k, C.c_longlong) for k in FIELDS]


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    so = str(d / "plan.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "plan.cpp")],
                   check=True)
    lib = C.CDLL(so)
    lib.replay.argtypes = [C.c_longlong, C.c_int, C.c_int, C.POINTER(C.c_longlong)]
    return lib


@pytest.fixture(scope="module")
def settle(plan):
    fn = plan.settle
    fn.restype = None
    fn.argtypes = [C.c_int, C.c_int, C.c_longlong, C.c_longlong, C.c_int, C.c_longlong, C.c_longlong, C.c_longlong,
                   C.POINTER(Out)]

    def call(block, sms, pixels, spp, tail_limit, path_limit):
        o = Out()
        resident = sms * 1024
        tail = min(pixels, 4 * resident, (1 << 26) // spp) if spp > 1 else 0
        fn(block, sms, resident, pixels, spp, tail, tail_limit, path_limit, C.byref(o))
        return o
    return call


ALL = 1 << 60
FRAMES = [(1280, 710), (1024, 768), (1600, 900), (1920, 1200), (4096, 2160), (1920, 1080), (777, 431), (512, 512),
          (552, 550), (451, 253), (1, 1), (7680, 4320)]


@pytest.mark.parametrize("sms", [148, 132, 1])
@pytest.mark.parametrize("tail_limit", [ALL, 0])
def test_slots_lie_in_the_buffer_asked_for(settle, sms, tail_limit):
    sizes = [w * h for w, h in FRAMES] + [10 ** 5 + 99991 * k for k in range(60)]
    for pixels in sizes:
        for spp in (1, 2, 3, 4, 5, 8, 13, 16, 64, 128, 512):
            o = settle(1024, sms, pixels, spp, tail_limit, ALL)
            what = (pixels, spp, {k: getattr(o, k) for k in FIELDS})
            assert o.path_bytes <= o.had_paths, what
            assert o.tail_bytes <= o.had_tail, what
            assert o.split + o.tail_pixels == pixels and o.items == o.split + o.tail_pixels * spp, what
            # no block without an item, none past the device's
            assert 1 <= o.grid <= sms and (o.grid - 1) * o.slots < o.items, what
            assert 32 <= o.slots <= 6 * 1024 and o.block == 1024, what


@pytest.mark.parametrize("tail_limit", [ALL, 0])
def test_a_frame_without_slots_takes_the_other_form(settle, tail_limit):
    for pixels in [w * h for w, h in FRAMES]:
        for spp in (1, 2, 16, 512):
            o, full = settle(1024, 148, pixels, spp, tail_limit, 0), settle(1024, 148, pixels, spp, tail_limit, ALL)
            assert (o.block, o.path_bytes, o.had_paths) == (128, 0, 0)
            assert (o.items, o.split, o.tail_pixels, o.tail_bytes) == (
                full.items, full.split, full.tail_pixels, full.tail_bytes)
            assert 1 <= o.slots <= 32 and 1 <= o.grid <= 148 * 4  # half the threads, in blocks of 128


@pytest.mark.parametrize("sms", [148, 132])
def test_replay_slots_and_vertices_lie_in_their_buffer(plan, sms):
    o = (C.c_longlong * 5)()
    for samples in [2048 * sms, 2048 * sms + 1, 10 ** 6, 3 * 10 ** 6 + 7, 512 * 512 * 32, 1920 * 1080 * 64, 1 << 33]:
        for depth in (3, 4, 6, 8, 13, 24, 32):
            plan.replay(samples, depth, sms, o)
            grid, slots, paths, vertices, used = o
            assert grid == sms and 32 <= slots <= 6 * 1024
            assert used <= paths and paths % 256 == 0
            assert vertices == grid * slots * depth * 32
            assert vertices <= (256 << 20) or slots <= 1024
            assert grid * slots <= samples + grid * 32
