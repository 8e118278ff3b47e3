"""The tests that drop a candidate for a whole tile of receivers, compiled for
the host and held against the per-receiver geometry in FP64 on random scenes:

* the diffraction shaft's near end holds the clamped stationary point of every
  receiver of the tile, also for a transmitter far along the edge's axis or
  close to it;
* a chain that the tile's bounds reject has no receiver whose FP64 back
  projection passes through every group's box;
* a triangle that closes a shaft cuts every segment between the near end and
  the tile.

Tolerance of the first: a triangle closes a shaft only with 1e-4 + 2e-5 M to
spare (M the largest coordinate 1-norm), so the near end may be off by half of
that.  The other two are exact statements."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from tests.test_utd_special_cpu import CSRC, CUDA_INCLUDE

# the device intrinsics that the header's kernels name, on the host
INTRINSICS = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include <cuda_runtime.h>
using std::isfinite;
using std::max;
using std::min;
#undef __launch_bounds__
#define __launch_bounds__(...)
struct Dim { int x = 0, y = 0, z = 0; };
static Dim threadIdx, blockIdx, blockDim;
template <typename T> static T __ldg(const T* p) { return *p; }
template <typename T> static T __shfl_sync(unsigned, T v, int) { return v; }
template <typename T> static T __shfl_xor_sync(unsigned, T v, int) { return v; }
template <typename T> static T __shfl_up_sync(unsigned, T v, int) { return v; }
static unsigned __ballot_sync(unsigned, bool v) { return v; }
static unsigned __reduce_add_sync(unsigned, unsigned v) { return v; }
static void __syncwarp() {}
static void __syncthreads() {}
static int __popc(unsigned v) { return __builtin_popcount(v); }
static int __ffs(unsigned v) { return __builtin_ffs(v); }
template <typename T, typename U> static T atomicAdd(T* p, U v) { T o = *p; *p += v; return o; }
template <typename T, typename U> static T atomicOr(T* p, U v) { T o = *p; *p |= v; return o; }
template <typename T, typename U> static T atomicMax(T* p, U v) { T o = *p; if (o < v) *p = v; return o; }
static float __int_as_float(int v) { float f; std::memcpy(&f, &v, 4); return f; }
static int __float_as_int(float v) { int f; std::memcpy(&f, &v, 4); return f; }
static double __longlong_as_double(long long v) { double f; std::memcpy(&f, &v, 8); return f; }
static float __fdividef(float a, float b) { return a / b; }
static float rsqrtf(float a) { return 1.f / std::sqrt(a); }
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static double __dmul_rn(double a, double b) { return a * b; }
static double __dsub_rn(double a, double b) { return a - b; }
"""

PROGRAM = INTRINSICS + r"""
#include "kernels.cuh"
using namespace wcb;

static std::mt19937_64 rng(5);
static double uni(double a, double b) { return a + (b - a) * std::generate_canonical<double, 53>(rng); }
static double lg(double a, double b) { return std::exp(uni(std::log(a), std::log(b))); }
static V3<double> vec(double s) { return v3(uni(-s, s), uni(-s, s), uni(-s, s)); }
static V3<double> unit(V3<double> v) { return v * (1.0 / length(v)); }
static V3<double> round32(V3<double> v) { return cast3<double>(cast3<float>(v)); }

// a tile's bounds (a point, a flat patch or a box) and receivers within them
static TileBounds tile(V3<double> at, double size, int kind) {
    const V3<float> p = cast3<float>(at);
    TileBounds b;
    const float c[3] = {p.x, p.y, p.z};
    for (int k = 0; k < 3; ++k) {
        b.lo[k] = c[k];
        b.hi[k] = kind == 0 || (kind == 1 && k == 2) ? c[k] : float(c[k] + uni(0.1, 1.0) * size);
    }
    return b;
}
static V3<double> inside(const TileBounds& b) {
    float r[3];
    for (int k = 0; k < 3; ++k) {
        const double f = std::min(std::max(uni(-0.3, 1.3), 0.0), 1.0);  // corners and faces among them
        r[k] = std::min(std::max(float(b.lo[k] + f * (double(b.hi[k]) - b.lo[k])), b.lo[k]), b.hi[k]);
    }
    return v3(double(r[0]), double(r[1]), double(r[2]));
}

static double shafts() {
    double worst = 0.0;
    for (int i = 0; i < 200000; ++i) {
        EdgeDev ed;
        std::memset(&ed, 0, sizeof(ed));
        const V3<double> c = round32(vec(lg(1.0, 3e3))), e = unit(vec(1.0)), side = unit(cross(e, vec(1.0)));
        const V3<double> bis = unit(cross(e, side));
        for (int k = 0; k < 3; ++k) {
            ed.pos[k] = k == 0 ? c.x : k == 1 ? c.y : c.z;
            ed.dir[k] = k == 0 ? e.x : k == 1 ? e.y : e.z;
            ed.bisector[k] = k == 0 ? bis.x : k == 1 ? bis.y : bis.z;
        }
        ed.half_length = lg(0.5, 300.0);
        SceneDev sc;
        std::memset(&sc, 0, sizeof(sc));
        sc.edges = &ed;
        // transmitters along the axis up to 1000 km away, on it up to 100 m off it
        const V3<double> S = round32(c + e * (lg(1.0, 1e6) * (i & 1 ? 1.0 : -1.0)) + side * (i % 3 ? lg(1e-7, 100.0) : 0.0));
        const V3<double> at = c + e * uni(-2.0, 2.0) * ed.half_length + unit(cross(e, vec(1.0))) * lg(1e-2, 200.0);
        const TileBounds b = tile(at, lg(0.1, 50.0), i % 4 < 2 ? 0 : i % 4 - 1);
        Shaft s;
        Ignore ig;
        edge_shaft(sc, 0, S, b, s, ig);
        double q[2];
        for (int k = 0; k < 2; ++k) q[k] = dot(cast3<double>(s.a[k]) - c, e);
        const double lo = std::min(q[0], q[1]), hi = std::max(q[0], q[1]);
        const V3<double> ds = S - c;
        const double ts = dot(ds, e), rs = length(ds - e * ts);
        for (int j = 0; j < 16; ++j) {
            const V3<double> dr = inside(b) - c;
            const double tr = dot(dr, e), rr = length(dr - e * tr);
            const double t_star = (rs + rr) > 0.0 ? ts + (tr - ts) * rs / (rs + rr) : ts;
            const double tc = std::fmin(std::fmax(t_star, -ed.half_length), ed.half_length);
            worst = std::max(worst, std::max(lo - tc, tc - hi) / (1e-4 + 2e-5 * double(s.size)));
        }
    }
    return worst;
}

static void chains(long long* rejected, long long* wrong) {
    constexpr int G = 4;
    *rejected = *wrong = 0;
    for (int i = 0; i < 60000; ++i) {
        const double at = i % 3 ? 0.0 : lg(10.0, 1e4);  // scenes far from the origin among them
        const V3<double> centre = vec(1.0) * at;
        const V3<double> S = round32(centre + vec(60.0)), R = centre + vec(80.0);
        const int d = 1 + i % 3;
        double planes[4 * 3], images[3 * 3];
        int groups[3];
        std::vector<float> box(6 * G);
        V3<double> img = S, n[3];
        for (int k = 0; k < d; ++k) {
            // planes that the next leg crosses more often than not
            n[k] = i & 1 ? unit(vec(1.0)) : v3(k % 2 ? 1.0 : 0.0, k % 2 ? 0.0 : 1.0, 0.0);
            const double hs = dot(n[k], img), hr = dot(n[k], R);
            const double off = std::max(hs, hr) + uni(-5.0, 40.0);
            img = img - n[k] * (2.0 * (hs - off));
            planes[4 * k] = n[k].x, planes[4 * k + 1] = n[k].y, planes[4 * k + 2] = n[k].z, planes[4 * k + 3] = off;
            images[3 * k] = img.x, images[3 * k + 1] = img.y, images[3 * k + 2] = img.z;
            groups[k] = k;
        }
        // boxes around R's own hits, up to past their edges
        V3<double> x = R;
        for (int k = d - 1; k >= 0; --k) {
            if (!back_project_step(x, planes, images, k)) x = x - n[k] * (dot(x, n[k]) - planes[4 * k + 3]);
            const double half = lg(0.5, 30.0), nc[3] = {n[k].x, n[k].y, n[k].z};
            const V3<double> o = vec(1.0) * (half * uni(0.0, 1.3)), c = x + o - n[k] * dot(o, n[k]);
            const double pc[3] = {c.x, c.y, c.z};
            for (int a = 0; a < 3; ++a) {
                const double ext = half * std::sqrt(std::max(1.0 - nc[a] * nc[a], 0.0)) + 1e-3;
                box[6 * k + a] = float(pc[a] - ext);
                box[6 * k + 3 + a] = float(pc[a] + ext);
            }
        }
        float4 pre[2] = {make_float4(float(planes[4 * (d - 1)]), float(planes[4 * (d - 1) + 1]),
                                     float(planes[4 * (d - 1) + 2]), float(planes[4 * (d - 1) + 3])),
                         make_float4(float(img.x), float(img.y), float(img.z), __int_as_float(groups[d - 1]))};
        MainParams p;
        std::memset(&p, 0, sizeof(p));
        p.sc.group_box = box.data();
        p.chain_planes = planes;
        p.chain_images = images;
        p.chain_groups = groups;
        p.chain_pre = pre;
        const TileBounds b = tile(R - vec(1.0) * (i % 7 ? lg(0.1, 5.0) : 0.0), lg(0.05, 15.0), i % 5 % 3);
        if (tile_may_reflect(p, b, 0, 0, d)) continue;
        ++*rejected;
        for (int j = 0; j < 64; ++j) {
            V3<double> x = inside(b);
            bool ok = true;
            for (int k = d - 1; k >= 0 && ok; --k) {
                ok = back_project_step(x, planes, images, k);
                const float* g = box.data() + 6 * groups[k];
                ok = ok && x.x >= g[0] && x.y >= g[1] && x.z >= g[2] && x.x <= g[3] && x.y <= g[4] && x.z <= g[5];
            }
            if (ok) {
                ++*wrong;
                break;
            }
        }
    }
}

static void triangles(long long* closed, long long* wrong) {
    *closed = *wrong = 0;
    for (int i = 0; i < 300000; ++i) {
        const V3<double> centre = i % 3 ? v3(0.0, 0.0, 0.0) : vec(lg(10.0, 1e4));
        Shaft s;
        const V3<double> a0 = round32(centre + vec(20.0)), a1 = round32(a0 + vec(i & 1 ? lg(0.1, 20.0) : 0.0));
        s.a[0] = cast3<float>(a0);
        s.a[1] = cast3<float>(a1);
        s.na = i & 1 ? 2 : 1;
        const TileBounds b = tile(centre + unit(vec(1.0)) * lg(20.0, 200.0), lg(0.1, 20.0), i % 5 % 3);
        s.size = 0.f;
        for (int k = 0; k < 3; ++k) s.lo[k] = b.lo[k], s.hi[k] = b.hi[k];
        const V3<float> lo = v3(b.lo[0], b.lo[1], b.lo[2]), hi = v3(b.hi[0], b.hi[1], b.hi[2]);
        s.size = std::max(std::max(norm1(lo), norm1(hi)) + norm1(hi - lo), std::max(norm1(s.a[0]), norm1(s.a[1])));
        s.side = 0.f;
        const V3<double> on = (a0 + a1) * 0.5 + ((cast3<double>(lo) + cast3<double>(hi)) * 0.5 - (a0 + a1) * 0.5) * uni(0.05, 0.95);
        const double half = lg(1.0, 300.0);
        const V3<double> u = unit(vec(1.0)), w = unit(cross(u, vec(1.0)));
        V3<float> t[3];
        for (int k = 0; k < 3; ++k) {
            const double ang = 2.0943951 * k + uni(-0.6, 0.6);
            t[k] = cast3<float>(on + (u * std::cos(ang) + w * std::sin(ang)) * half);
        }
        if (!triangle_cuts_shaft(s, t[0], t[1], t[2])) continue;
        ++*closed;
        const V3<double> v0 = cast3<double>(t[0]), v1 = cast3<double>(t[1]), v2 = cast3<double>(t[2]);
        const V3<double> n = cross(v1 - v0, v2 - v0);
        for (int j = 0; j < 32; ++j) {
            const V3<double> p0 = a0 + (a1 - a0) * (j & 1 ? uni(0.0, 1.0) : double((j >> 1) & 1)), p1 = inside(b);
            const double h0 = dot(n, p0 - v0), h1 = dot(n, p1 - v0);
            const V3<double> x = p0 + (p1 - p0) * (h0 / (h0 - h1));
            const bool in = dot(cross(v1 - v0, x - v0), n) > 0 && dot(cross(v2 - v1, x - v1), n) > 0 &&
                            dot(cross(v0 - v2, x - v2), n) > 0;
            if (h0 * h1 >= 0 || !in) {
                ++*wrong;
                break;
            }
        }
    }
}

int main() {
    std::printf("shaft %.6g\n", shafts());
    long long n, bad;
    chains(&n, &bad);
    std::printf("chains %lld %lld\n", n, bad);
    triangles(&n, &bad);
    std::printf("triangles %lld %lld\n", n, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def output(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("reject")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-D__noinline__=", f"-I{CUDA_INCLUDE}", f"-I{CSRC}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: [float(t) for t in line.split()[1:]] for line in out.splitlines()}


def test_shaft_holds_every_stationary_point(output):
    assert output["shaft"][0] <= 0.5


def test_rejected_chains_have_no_path(output):
    rejected, wrong = output["chains"]
    assert rejected > 10000
    assert wrong == 0


def test_closing_triangles_cut_every_segment(output):
    closed, wrong = output["triangles"]
    assert closed > 3000
    assert wrong == 0
