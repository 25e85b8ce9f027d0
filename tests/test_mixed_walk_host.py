"""The mixed solve's walk over matrix slices (SliceWalk), its own text on the CPU
with copies that the test delivers or holds back.  A slice's columns and values
are copied into a stage while the slice before it is worked on; when a copy does
not arrive the walk has to end there: nothing of the stage is read, no other
copy is started into it, by this walk or the warp's next one, and the one
outstanding is left to be awaited once more.  Nothing of this can be asked of a
GPU, where a copy arrives."""

import ctypes as C

import numpy as np
import pytest

import host_kernel as hk

CODE = r"""
#include <limits>
constexpr int kSlice = 32;
constexpr int32_t kPad = -1;
constexpr int16_t kPad16 = std::numeric_limits<int16_t>::min();
template <class T> static inline T __ldcs(const T* p) { return *p; }
static inline float ldv(const float* p) { return *p; }
static int __all_sync(unsigned, bool v) { return v; }
// the barrier: phases completed, and the copies that fill the stage when awaited
static int waits, copies, reads, lose_at, torn;
static bool open_phase;
static struct { void* dst; const void* src; unsigned bytes; } queue[2];
static int queued;
static void bulk_expect(uint64_t*, unsigned) {
  torn += open_phase;  // a copy into a stage whose last one is outstanding
  open_phase = true;
  ++copies;
}
static void bulk_copy(void* dst, const void* src, unsigned bytes, uint64_t*) {
  if (queued < 2) queue[queued++] = {dst, src, bytes};
}
static unsigned phase;
static bool bulk_wait(uint64_t*, unsigned parity) {
  ++waits;
  if (parity != phase) return true;  // that phase is over
  if (!open_phase || waits == lose_at) return false;
  for (int k = 0; k < queued; ++k) std::memcpy(queue[k].dst, queue[k].src, queue[k].bytes);
  queued = 0;
  open_phase = false;
  phase ^= 1u;
  return true;
}
%s
static float stage[4096];
// two walks of one warp (the matrix twice) over ns slices, lane `lane`
extern "C" int walk(int ns, int n, const int32_t* soff, const int32_t* sw, const int32_t* col,
                    const float* val, int lane, int lose, float* y, int* info) {
  waits = copies = reads = queued = torn = 0;
  lose_at = lose;
  open_phase = false;
  phase = 0;
  threadIdx.x = 0;  // lane 0 makes the copies; the row's lane is added to the pointers
  uint64_t mb = 0;
  int4 places[1];
  int bad = 0;
  unsigned st = 0;
  using W = SliceWalk<Cols32, float, 4>;
  W a{soff, sw, Cols32{col}, val, reinterpret_cast<char*>(stage), 0, ns, 0, 0, 0, 0, places, &mb,
      &bad};
  W b = a;
  places[0] = a.first_two(0);
  int rows = 0;
  a.start(0, st);
  for (W* w : {&a, &b}) {
    if (w == &b) b.start(0, st);
    while (w->s < ns) {
      const int32_t s = w->s, i = s * kSlice;
      const float t = w->row(i, [&](int32_t c) {
        ++reads;
        if (c < 0 || c >= n) return std::nanf("");
        return float(c + 1);
      }, [] {}, st);
      y[rows++] = t;
    }
  }
  info[0] = waits, info[1] = copies, info[2] = reads, info[3] = bad, info[4] = torn;
  info[5] = (st & kWalkPending) != 0, info[6] = (st & kWalkPhase) == phase;
  return rows;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    text = hk.source("xg_cg.cu")
    piece = hk.cut(text, "Cols32", "kMixThreads", "kMixRound", "kWalkPhase", "SliceWalk")
    # one warp takes every slice
    piece = piece.replace("kMixThreads / 32;", "1;")
    return hk.build(tmp_path_factory.mktemp("walk"), CODE % piece)


def _matrix(ns, seed):
    """Slices of 0 to 7 entries a row (up to 4 are staged), row 0 of each filled."""
    rng = np.random.default_rng(seed)
    sw = rng.integers(0, 8, ns).astype(np.int32)
    soff = np.concatenate([[0], np.cumsum(sw * 32)]).astype(np.int32)
    col = np.full(max(1, soff[-1]), -1, np.int32)
    val = np.zeros(col.size, np.float32)
    for s in range(ns):
        for k in range(sw[s]):
            if rng.random() < 0.8:
                col[soff[s] + k * 32] = rng.integers(0, ns * 32)
            val[soff[s] + k * 32] = rng.integers(1, 9)
    return soff, sw, col, val


def _run(lib, ns, m, lose):
    y, info = np.zeros(2 * ns + 4, np.float32), np.zeros(7, np.int32)
    p = [a.ctypes.data_as(C.c_void_p) for a in m]
    rows = lib.walk(ns, ns * 32, *p, 0, lose, y.ctypes.data_as(C.c_void_p),
                    info.ctypes.data_as(C.c_void_p))
    return y[:rows], info


@pytest.mark.parametrize("seed", range(6))
def test_walk(lib, seed):
    ns = 9
    soff, sw, col, val = m = _matrix(ns, seed)
    e = [soff[s] + 32 * np.arange(sw[s]) for s in range(ns)]
    want = np.array([sum(float(v) * (c + 1) for c, v in zip(col[k], val[k]) if c >= 0) for k in e])
    y, (waits, copies, reads, bad, torn, pending, _) = _run(lib, ns, m, 0)
    filled = int((sw > 0).sum())
    assert np.array_equal(y, np.concatenate([want, want]))
    assert (waits, copies, bad, torn, pending) == (2 * filled, 2 * filled, 0, 0, 0)
    for lose in range(1, 2 * filled + 1):
        y, (waits, copies, reads, bad, torn, pending, phase) = _run(lib, ns, m, lose)
        assert bad == 1 and torn == 0
        assert waits == copies == lose  # no wait and no copy after the lost one
        assert pending and phase  # and that one can still be awaited
        slices = np.flatnonzero(sw)
        done = [slices[k % filled] for k in range(lose - 1)]
        assert len(y) == (lose > filled) * ns + slices[(lose - 1) % filled] + 1
        assert y[-1] == 0  # nothing of the stage was read
        beyond = [int((col[e[s]][4:] >= 0).sum()) for s in done]
        assert reads == sum(min(sw[s], 4) for s in done) + sum(beyond)
