"""A warp's list of sample pairs (warp_pairs, describe.cu), checked on the CPU:
the function's own text, compiled with the warp's 32 lanes as threads. A plain
store to the row starts becomes visible to the other lanes at the lane's next
__syncwarp and no earlier, as a shuffle or a ballot does not order memory, and
the memory holds other bits before. Every sample inside the rotated square is
in exactly one pair."""
import shutil
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "sift_wgpu_gb300" / "csrc"

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <set>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
#define __align__(n) alignas(n)
using std::max;
using std::min;
constexpr int kDescRadGrid = 31;
std::barrier<> together(32);
thread_local int me;
thread_local std::vector<std::pair<uint32_t*, uint32_t>> stores;
struct Word {
    uint32_t v;
    void operator=(uint32_t x) { stores.emplace_back(&v, x); }
};
float rcp_approx(float x) { return 1.0f / x; }
int floor_i(float x) { return (int)std::floor(x); }
int __popc(uint32_t x) { return __builtin_popcount(x); }
void atomicOr(Word* w, uint32_t x) { __atomic_fetch_or(&w->v, x, __ATOMIC_SEQ_CST); }
void __syncwarp() {
    for (auto& s : stores) *s.first = s.second;
    stores.clear();
    together.arrive_and_wait();
}
int lanes[32];
int exchange(int v, int from) {
    lanes[me] = v;
    together.arrive_and_wait();
    const int r = lanes[from];
    together.arrive_and_wait();
    return r;
}
int __shfl_up_sync(uint32_t, int v, int d, int width) { return exchange(v, me % width >= d ? me - d : me); }
int __shfl_sync(uint32_t, int v, int from) { return exchange(v, from); }
uint32_t __ballot_sync(uint32_t, bool p) {
    static uint32_t bits;
    lanes[me] = p;
    together.arrive_and_wait();
    uint32_t b = 0;
    for (int i = 0; i < 32; ++i) b |= (uint32_t)lanes[i] << i;
    together.arrive_and_wait();
    return b;
}
"""

MAIN = r"""
int main() {
    int bad = 0, checked = 0;
    for (int rad : {1, 2, 7, 15, 16, 22, 31})
        for (int a = 0; a < 9; ++a) {
            const float ang = a == 8 ? 1e-6f : -3.1f + 0.77f * a, ca = std::cos(ang), sa = std::sin(ang);
            const float lim = rad * 0.88388f;  // 2.5 cells of a window of 4 whose diagonal is 2 rad
            const int gst = 2 * rad + 4;
            std::set<std::pair<int, int>> seen;
            for (int warp = 0; warp < 4; ++warp) {
                WarpPairs w;
                std::memset((void*)&w, 0xa5, sizeof w);
                int n[32];
                std::vector<std::thread> lane;
                for (int l = 0; l < 32; ++l)
                    lane.emplace_back([&, l] {
                        me = l;
                        n[l] = warp_pairs(&w, ca, sa, lim, rad, gst, warp, l);
                    });
                for (auto& t : lane) t.join();
                int row = -1;
                for (int m = 0; m < n[0]; ++m) {
                    row += w.start[m >> 5].v >> (m & 31) & 1u;
                    if (row < 0 || row >= kWarpRows) return printf("row %d\n", row), 1;
                    const int px = (int)w.row[row].px + 2 * m, py = (int)w.row[row].py;
                    bad += !seen.insert({px, py}).second || std::abs(py) > rad || px < -rad - 1 || px > rad;
                }
            }
            for (int y = -rad; y <= rad; ++y)
                for (int x = -rad; x <= rad; ++x) {
                    if (!(std::fabs(ca * x + sa * y) < lim && std::fabs(ca * y - sa * x) < lim)) continue;
                    // pairs start at even distances from -rad - parity of the grid row
                    const int first = -rad - ((y + rad + 1) & 1), px = x - ((x - first) & 1);
                    bad += !seen.count({px, y});
                    ++checked;
                }
        }
    printf("%d checked, %d bad\n", checked, bad);
    return bad || checked < 10000;
}
"""


def test_every_sample_is_in_one_pair(tmp_path):
    src = (CSRC / "describe.cu").read_text()
    text = src[src.index("struct __align__(16) PairRow"):src.index("// The eight shares of a sample")]
    assert "uint32_t start[kWarpWords]" in text
    (tmp_path / "p.cpp").write_text(SHIM + text.replace("uint32_t start[kWarpWords]", "Word start[kWarpWords]") + MAIN)
    subprocess.run([shutil.which("g++"), "-std=c++20", "-O1", "-ffp-contract=off", "-pthread", "-o", tmp_path / "p",
                    tmp_path / "p.cpp"], check=True)
    r = subprocess.run([tmp_path / "p"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
