"""The warp routine's shared-memory accesses under ThreadSanitizer: the code of
csrc/quadrature.cuh itself, compiled for the host with its 32 lanes as threads.
__syncwarp orders memory between the lanes; shuffles, reductions and votes
exchange registers and order nothing (their stand-ins use relaxed atomics only,
which the sanitizer does not take for synchronisation), so two lanes touching
one word of the panel list without a __syncwarp between them are reported."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "options-pricing-engine-rs_b200", "csrc")

# Stand-ins: a peaked integrand for the node evaluation (what matters is the
# order in which panels are bisected; the peak's place is the integral's x).
CF_STUB = r"""
#pragma once
namespace ope {
struct CfConsts { double x; };
struct NodeCf { double w, a, u; };
template <bool BATES> inline NodeCf node_cf(const CfConsts&, double t) { return {1.0, 0.0, t}; }
inline double node_u_of(double t) { return t; }
inline double node_finish(double x, double u, double, double w) {
    return w * (0.001 / ((u - x) * (u - x) + 1e-6) + 0.3 * std::sin(40.0 * u));
}
}
"""
CHECKED_STUB = r"""
#pragma once
#define ope_check(cond, code) (cond)
"""
MAIN = r"""
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#define __device__
#define __constant__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
using std::max;
using std::min;
struct double2 { double x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline long long __double_as_longlong(double a) { long long r; std::memcpy(&r, &a, 8); return r; }
inline double __longlong_as_double(long long a) { double r; std::memcpy(&r, &a, 8); return r; }
inline double2 __ldcg(const double2* p) { return *p; }
inline void __stcg(double2* p, double2 v) { *p = v; }

static thread_local int t_lane;
// a barrier that makes every lane wait, in terms of memory order `o`
static std::atomic<unsigned> g_in[2], g_turn[2];
static void meet(int which, std::memory_order up, std::memory_order down) {
    const unsigned turn = g_turn[which].load(std::memory_order_relaxed);
    if (g_in[which].fetch_add(1, up) == 31) {
        g_in[which].store(0, std::memory_order_relaxed);
        g_turn[which].store(turn + 1, down);
    } else {
        while (g_turn[which].load(up == std::memory_order_relaxed ? up : std::memory_order_acquire) == turn)
            std::this_thread::yield();
    }
}
inline void __syncwarp() { meet(0, std::memory_order_acq_rel, std::memory_order_release); }
inline void converge() { meet(1, std::memory_order_relaxed, std::memory_order_relaxed); }
static std::atomic<uint64_t> g_slot[32];
template <class T> inline T exchange(T v, int from) {
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof(T));
    g_slot[t_lane].store(b, std::memory_order_relaxed);
    converge();
    b = g_slot[from].load(std::memory_order_relaxed);
    converge();
    std::memcpy(&v, &b, sizeof(T));
    return v;
}
template <class T> inline T __shfl_xor_sync(unsigned, T v, int m) { return exchange(v, t_lane ^ m); }
template <class F> inline unsigned reduce(unsigned v, F f) {
    unsigned r = exchange(v, t_lane ^ 0);
    for (int m = 1; m < 32; m <<= 1) r = f(r, exchange(r, t_lane ^ m));
    return r;
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
    return reduce(v, [](unsigned a, unsigned b) { return a > b ? a : b; });
}
inline int __any_sync(unsigned, int v) { return (int)reduce(v != 0, [](unsigned a, unsigned b) { return a | b; }); }

#include "quadrature.cuh"

using namespace ope;
static PanelStore L;
static uint8_t g_child[kRunLinks], g_slots[kMaxPanels];
static double2 g_wa[kRunEntries * 16];
static CfConsts g_c;
static double g_total[32][2][4];
static int g_nbis[2][4];

template <bool CACHED> static void lanes(int k, double x, double tol) {
    std::vector<std::thread> ts;
    g_c.x = x;
    for (int lane = 0; lane < 32; ++lane)
        ts.emplace_back([=] {
            t_lane = lane;
            const LaneRule R = lane_rule(lane);
            RunCacheWarp rc{g_wa, g_child, g_slots, 63, 0};
            if (CACHED && lane == 0) g_child[kNoEntry] = (uint8_t)kNoEntry;
            __syncwarp();
            for (int again = 0; again < (CACHED ? 2 : 1); ++again) {  // the second reads what the first has stored
                int nb = 0;
                const double v = gk_integrate_warp<false, CACHED>(g_c, tol, L, lane, R, &nb, NoTrace(), &rc);
                g_total[lane][CACHED][k] = v;
                if (lane == 0) g_nbis[CACHED][k] = nb;
                __syncwarp();
            }
        });
    for (auto& t : ts) t.join();
}

int main() {
    // peaks at the left end, inside, at the right end; the last one runs into the panel limit
    const double xs[4] = {1e-3, 0.37, 0.999, 0.5}, tols[4] = {1e-7, 1e-7, 1e-7, -1.0};
    for (int k = 0; k < 4; ++k) {
        lanes<false>(k, xs[k], tols[k]);
        lanes<true>(k, xs[k], tols[k]);
        if (g_total[0][0][k] != g_total[0][1][k] || g_nbis[0][k] != g_nbis[1][k]) return 2;
        std::printf("%d bisections, integral %.15g\n", g_nbis[0][k], g_total[0][0][k]);
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
def test_no_two_lanes_race_on_the_panel_list(tmp_path):
    shutil.copy(os.path.join(CSRC, "quadrature.cuh"), tmp_path / "quadrature.cuh")
    (tmp_path / "cf_device.cuh").write_text(CF_STUB)
    (tmp_path / "checked.cuh").write_text(CHECKED_STUB)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "race")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-ffp-contract=off", "-fsanitize=thread", "-pthread",
                    "-Wno-attributes", str(tmp_path / "main.cpp"), "-o", exe], check=True, cwd=tmp_path)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, TSAN_OPTIONS="halt_on_error=0:exitcode=66:history_size=7"))
    races = sorted(set(re.findall(r"quadrature\.cuh:(\d+)", r.stderr)))
    assert r.returncode == 0 and not races, (r.returncode, races, r.stderr[:3000])
    assert [int(v) for v in re.findall(r"(\d+) bisections", r.stdout)][-1] == 199
