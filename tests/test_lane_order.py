"""The step's shared-memory traffic between the lanes of a one-warp column
(32 levels or fewer) is ordered by synchronisation: shuffles and votes make
lanes wait for one another but order no memory accesses.

The step body of csrc/mp_kernel.cuh runs here on the host, one thread per
lane, under ThreadSanitizer. A warp barrier is a barrier the sanitizer knows;
a shuffle or a vote exchanges its values through relaxed atomics, which order
nothing. A shared value that one lane writes and another reads, with only
shuffles between, is then reported as a data race. The outputs are compared
with the oracle, so that the run is the step and not a part of it."""
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyshield_b200", "csrc")

SOURCE = r"""
#include <pthread.h>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <string>
#include <thread>
#include <vector>
using std::min;
using std::max;
using std::isfinite;

// ------------------------------------------------------- a warp of threads
static thread_local int lane_id;
static pthread_barrier_t warp_barrier;
static std::atomic<unsigned long long> box[2][32];
static std::atomic<unsigned long long> arrivals{0};
static thread_local unsigned long long generation;

static void exchange(unsigned long long mine, unsigned long long (&all)[32]) {
  const unsigned long long g = generation++;
  box[g & 1][lane_id].store(mine, std::memory_order_relaxed);
  arrivals.fetch_add(1, std::memory_order_relaxed);
  while (arrivals.load(std::memory_order_relaxed) < 32 * (g + 1)) std::this_thread::yield();
  for (int l = 0; l < 32; ++l) all[l] = box[g & 1][l].load(std::memory_order_relaxed);
}
template <class T>
static T from_lane(T x, int src) {
  unsigned long long mine = 0, all[32];
  std::memcpy(&mine, &x, sizeof(T));
  exchange(mine, all);
  std::memcpy(&x, &all[src >= 0 && src < 32 ? src : lane_id], sizeof(T));
  return x;
}
template <class T> T __shfl_sync(unsigned, T x, int l) { return from_lane(x, l); }
template <class T> T __shfl_up_sync(unsigned, T x, int d) { return from_lane(x, lane_id - d); }
template <class T> T __shfl_down_sync(unsigned, T x, int d) { return from_lane(x, lane_id + d); }
template <class T> T __shfl_xor_sync(unsigned, T x, int m) { return from_lane(x, lane_id ^ m); }
static unsigned __ballot_sync(unsigned, bool p) {
  unsigned long long all[32];
  exchange(p, all);
  unsigned r = 0;
  for (int l = 0; l < 32; ++l) r |= (all[l] ? 1u : 0u) << l;
  return r;
}
static bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
static int __reduce_min_sync(unsigned, int v) {
  unsigned long long all[32];
  exchange((unsigned)v, all);
  for (int l = 0; l < 32; ++l) v = min(v, (int)(unsigned)all[l]);
  return v;
}
static void __syncwarp() { pthread_barrier_wait(&warp_barrier); }
static void __syncthreads() { pthread_barrier_wait(&warp_barrier); }
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static double __dadd_rn(double a, double b) { return a + b; }
static int atomicCAS(int* p, int want, int v) {
  __atomic_compare_exchange_n(p, &want, v, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED);
  return want;
}
struct Dim { int x; };
static thread_local Dim threadIdx;
struct cudaStream;
typedef cudaStream* cudaStream_t;
typedef int cudaError_t;

#include "kernel_head.cuh"
#include "mp_setup.h"

using namespace shield;
using LY = ColumnLayout<1, 1>;

int main(int argc, char** argv) {
  // configuration, step length and levels; then the 13 fields of one column, land, area
  FILE* f = fopen(argv[1], "rb");
  ShieldMpConfig cfg;
  double dt;
  int L;
  if (fread(&cfg, sizeof cfg, 1, f) != 1 || fread(&dt, sizeof dt, 1, f) != 1 || fread(&L, sizeof L, 1, f) != 1) return 2;
  std::vector<double> in(13 * L + 2), qaz(L, 0.0);
  if (fread(in.data(), sizeof(double), in.size(), f) != in.size()) return 2;
  fclose(f);
  static MpArgs A;
  setupm(cfg, A.K);
  std::string why;
  if (set_timestep(cfg, A.K, dt, why) != 0) return 3;
  A.KF = to_float(A.K);
  A.nx = A.ny = 1;
  A.nz = L;
  A.ncol = 1;
  for (int n = 0; n < 13; ++n) A.in[n] = Fld3{in.data() + n * L, 1, 1, 1};
  A.in[IN_QAZ] = Fld3{qaz.data(), 1, 1, 1};
  A.land = Fld2{in.data() + 13 * L, 1, 1};
  A.area = Fld2{in.data() + 13 * L + 1, 1, 1};
  double rain = 0.0;
  int err = 0;
  A.rain = &rain;
  A.err = &err;
  A.by_nx = fast_div(1);
  std::vector<double> sm(Smem<LY>::total, std::numeric_limits<double>::quiet_NaN());
  for (int n = 0; n < N_IN; ++n)
    for (int k = 0; k < L; ++k) sm[n * LY::RP + k] = A.in[n].p[k];
  pthread_barrier_init(&warp_barrier, nullptr, 32);
  std::vector<std::thread> warp;
  for (int l = 0; l < 32; ++l)
    warp.emplace_back([&, l] {
      lane_id = l;
      threadIdx.x = l;
      mp_body<LY, false>(A, sm.data(), sm.data() + Smem<LY>::scratch, sm.data() + Smem<LY>::work, 0);
    });
  for (auto& t : warp) t.join();
  for (int o = 0; o < N_OUT; ++o)
    for (int k = 0; k < L; ++k) std::printf("%.17g\n", sm[o * LY::RP + k]);
  std::printf("%.17g %d\n", rain, err);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("lanes")
    head = open(os.path.join(CSRC, "mp_kernel.cuh")).read()
    body = head[:head.index("template <class LY, int MINB, bool MIXED, bool FLAGS = false>\n__global__")]
    (tmp / "kernel_head.cuh").write_text(body + "\n}\n}\n")
    (tmp / "t.cpp").write_text(SOURCE)
    (tmp / "empty.cpp").write_text("int main() { return 0; }")
    flags = ["g++", "-O1", "-g", "-std=c++17", "-w", "-pthread", "-fsanitize=thread", "-ffp-contract=off"]
    if subprocess.run(flags + [str(tmp / "empty.cpp"), "-o", str(tmp / "empty")], capture_output=True).returncode or \
            subprocess.run([str(tmp / "empty")], capture_output=True).returncode:
        pytest.skip("no ThreadSanitizer on this host")
    r = subprocess.run(flags + ["-I", CSRC, "-I", os.path.join(os.path.dirname(os.path.dirname(CSRC)), "include"), "-I",
                                str(tmp), str(tmp / "t.cpp"), "-o", str(tmp / "t")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return tmp


@pytest.mark.parametrize("borrow", [False, True])
@pytest.mark.parametrize("fix_negative", [True, False])
def test_no_unordered_access(program, fix_negative, borrow):
    from golden_io import MP_TENDENCIES
    from oracle.microphysics import OracleMicrophysics
    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200._lib import MP_STATE_FIELDS, make_config
    from pyshield_b200.inputs import make_state

    from mp_helpers import TOL_PLAIN, gpu_floors

    L, dt = 31, 225.0
    cfg = PhysicsConfig(dt_atmos=dt, fix_negative=fix_negative)
    state, area = make_state(1, L, seed=12, n_cube=12, sat_fraction=0.1)
    if borrow:
        state["qvapor"][[3, 9, 10, L - 1]] = [[-1e-5], [-2e-5], [1e-6], [-1e-6]]
    data = np.concatenate([np.concatenate([state[n][:, 0] for n in MP_STATE_FIELDS]), state["land"], area])
    path = program / "in.bin"
    path.write_bytes(bytes(make_config(cfg)) + np.float64(dt).tobytes() + np.int32(L).tobytes() + data.tobytes())
    r = subprocess.run([str(program / "t"), str(path)], capture_output=True, text=True,
                       env={**os.environ, "TSAN_OPTIONS": "exitcode=66 halt_on_error=0"}, timeout=600)
    assert "WARNING: ThreadSanitizer" not in r.stderr, r.stderr[:3000]
    assert r.returncode == 0, r.stderr[:3000]
    if not fix_negative and borrow:
        return  # negative vapour unmended: the reference's expressions take logs of it
    out = np.array(r.stdout.split(), dtype=float)
    got = out[:-2].reshape(-1, L)
    mp = OracleMicrophysics(cfg, 1, L, area)
    mp(state, dt)
    floors = gpu_floors(state, {n: state[n] for n in MP_TENDENCIES}, dt)
    for n, v in zip(MP_TENDENCIES + ("wmp",), got):
        ref = state[n][:, 0]
        tol = TOL_PLAIN * np.max(np.abs(ref)) + floors.get(n, 0.0)
        assert np.max(np.abs(v - ref)) <= tol, (n, np.max(np.abs(v - ref)), tol)
