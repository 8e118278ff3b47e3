"""Special functions and closed-form Jacobians of the UTD, compiled for the host.

* the KP transition function and the Fresnel complement (FP64 and FP32) against
  the Faddeeva function, across the ends of the pole term and of the
  large-argument expansion;
* the closed-form Jacobians of a mended KP term and of a half-space face factor
  against the same templates evaluated with dual-number lanes;
* the reverse mode of a reflection record against dual lanes of the same chain.

Tolerances: F and the complement come from a sum of positive terms and one
division each, so a few FP64 (FP32) roundings: 4e-15 (1e-6, FP32 including the
rounding of the phase, up to 2 pi, 4e-7), where the FP64 expansion from x = 400
drops a term of 4e-14.  A Jacobian differs from the dual lanes by rounding
alone, amplified by the cancellation in F' = F (1/(2x) + j) - j, at most 2x / |F'| / x
~ 1e4 ulp for x < 400 and up to 1e-7 relative on the far side, where F' itself is
a difference of O(1) numbers around 1e-6: 1e-9 of the term's scale.  A reflection
record's gradient carries the conditioning of its images (a grazing line's
1 / (e.n), up to 1e3 per bounce and cubed over three, on 1e-16): 1e-7 of the
derivative's own modulus.
"""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
from scipy.special import wofz

CSRC = Path(__file__).resolve().parents[1] / "witwin_channel_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
using std::isfinite;
#include "reflection_adjoint.cuh"
using namespace wcb;

static double worst(Cx<double> got, double re, double im, double scale) {
    return std::max(std::fabs(got.re - re), std::fabs(got.im - im)) / scale;
}

// The record's field with every input a dual lane: S, R (3 each), per plane
// normal (3), offset, eps_r, sigma_e, then the frequency.
constexpr int kDepth = 3, kLanes = 7 + 6 * kDepth;
using DL = Dual<kLanes>;
static Cx<DL> dual_reflection(const ReflectionRecordIn<kDepth>& in, double sq) {
    int lane = 0;
    auto var = [&](double v) { DL x(v); x.d[lane++] = 1.0; return x; };
    auto var3 = [&](V3<double> v) { const DL a = var(v.x), b = var(v.y), c = var(v.z); return v3(a, b, c); };
    auto con3 = [&](V3<double> v) { return v3(DL(v.x), DL(v.y), DL(v.z)); };
    const V3<DL> S = var3(in.S), R = var3(in.R), ez = v3(DL(0.0), DL(0.0), DL(1.0));
    V3<DL> n[kDepth], img[kDepth], hit[kDepth];
    DL off[kDepth];
    Slab<DL> slab[kDepth];
    const int d = in.depth;
    for (int q = 0; q < d; ++q) {
        n[q] = var3(in.n[q]);
        off[q] = var(in.off[q]);
        const DL e = var(in.slab[q].eps_r), g = var(in.slab[q].sigma_e);
        slab[q] = Slab<DL>{e, g, DL(in.slab[q].mu_r), DL(in.slab[q].gain), DL(in.slab[q].thickness)};
    }
    const DL f = var(in.f), k = f * (kTwoPi / kC0), wl = DL(kC0) / f;
    V3<DL> p = S;
    for (int q = 0; q < d; ++q) {
        p = p - n[q] * (DL(2.0) * (dot(p, n[q]) - off[q]));
        img[q] = p;
    }
    V3<DL> x = R;
    for (int q = d - 1; q >= 0; --q) {
        x = x + (img[q] - x) * ((off[q] - dot(x, n[q])) / dot(img[q] - x, n[q]));
        hit[q] = x;
    }
    const DL L = length(R - p);
    V3<DL> prev = S, outgoing = safe_normalize(hit[0] - prev, ez);
    C3<DL> value = c3_from_real(transverse(outgoing, con3(in.tx_pol)));
    for (int q = 0; q < d; ++q) {
        const V3<DL> inc = safe_normalize(hit[q] - prev, outgoing);
        reflect_bounce(value, outgoing, inc, n[q], slab[q], f, wl);
        prev = hit[q];
    }
    const V3<DL> dir = safe_normalize(R - prev, outgoing);
    value = c3_scale(value, phasor_neg_kd(k, L) * (DL(1.0) / (DL(2.0) * k * s_max(L, kUtdEps))));
    return project_receiver(value, dir, con3(in.rx_pol)) * DL(sq);
}

int main() {
    // special functions: lines "x F.re F.im c.re c.im F32.re F32.im c32.re c32.im"
    for (int i = 0; i < 4000; ++i) {
        const double x = std::pow(10.0, -8.0 + 11.5 * i / 3999.0);
        const float xf = float(x);
        const Cx<double> F = transition<double>(x), c = fresnel_pos<double>(x).complement(x, fresnel_phasor<double>(x));
        const Cx<float> G = transition<float>(xf), d = fresnel_pos<float>(xf).complement(xf, fresnel_phasor<float>(double(xf)));
        std::printf("%.17g %.17g %.17g %.17g %.17g %.9g %.9g %.9g %.9g\n", x, F.re, F.im, c.re, c.im, G.re, G.im, d.re, d.im);
    }
    std::mt19937_64 rng(3);
    auto uni = [&](double a, double b) { return a + (b - a) * std::generate_canonical<double, 53>(rng); };
    double term = 0.0, face = 0.0;
    for (int i = 0; i < 200000; ++i) {
        const double n = uni(1.05, 2.0), phi_p = uni(0.0, n * kPi);
        double phi = uni(0.0, n * kPi);
        if (i % 7 == 0) phi = n * kPi;                          // a receiver clamped onto face n
        if (i % 5 == 0) phi = std::min(phi_p + kPi + uni(-1e-3, 1e-3), n * kPi);  // a shadow boundary
        const double kl = std::pow(10.0, uni(-1.0, 5.0)), t = uni(0.0, 1.0), g = uni(0.0, 1.0);
        const bool incident = i & 1;
        const int s = (i >> 1) & 1 ? 1 : -1;
        const double beta = incident ? phi - phi_p : phi + phi_p;
        Dual<5> b(beta), d2(n), d3(kl), d4(t), d5(g);
        b.d[0] = d2.d[1] = d3.d[2] = d4.d[3] = d5.d[4] = 1.0;
        const Cx<Dual<5>> want = mended_term(b, d2, d3, d4, d5, s, incident);
        const MendedJet got = mended_jet(beta, n, kl, t, g, s, incident);
        const Cx<double> lanes[5] = {got.db, got.dn, got.dkl, got.dt, got.dg};
        const double v = std::hypot(want.re.v, want.im.v) + 1.0;
        term = std::max(term, worst(got.v, want.re.v, want.im.v, v));
        for (int l = 0; l < 5; ++l)
            term = std::max(term, worst(lanes[l], want.re.d[l], want.im.d[l],
                                        std::hypot(want.re.d[l], want.im.d[l]) + v * (l == 2 ? 1.0 / kl : 1.0)));
        const Slab<double> m{uni(1.0, 12.0), std::pow(10.0, uni(-4.0, 1.0)), 1.0, uni(0.5, 1.0), 0.2};
        const double ang = uni(-0.5, 2.0) * kPi, f = std::pow(10.0, uni(8.0, 11.0));
        Dual<4> a4(ang), e4(m.eps_r), s4(m.sigma_e), f4(f);
        a4.d[0] = e4.d[1] = s4.d[2] = f4.d[3] = 1.0;
        const Slab<Dual<4>> md{e4, s4, Dual<4>(m.mu_r), Dual<4>(m.gain), Dual<4>(m.thickness)};
        Cx<Dual<4>> te, tm;
        halfspace_fresnel(s_sin(a4), md, f4, &te, &tm);
        FaceJet fj;
        face_jet(ang, m, f, fj);
        face = std::max(face, std::max(worst(fj.te, te.re.v, te.im.v, 1.0), worst(fj.tm, tm.re.v, tm.im.v, 1.0)));
        for (int l = 0; l < 4; ++l) {
            const double sc[4] = {1.0, 1.0, 1.0 / m.sigma_e, 1.0 / f};
            face = std::max(face, worst(fj.dte[l], te.re.d[l], te.im.d[l], std::hypot(te.re.d[l], te.im.d[l]) + sc[l]));
            face = std::max(face, worst(fj.dtm[l], tm.re.d[l], tm.im.d[l], std::hypot(tm.re.d[l], tm.im.d[l]) + sc[l]));
        }
    }
    double refl = 0.0;
    for (int i = 0; i < 20000; ++i) {
        ReflectionRecordIn<kDepth> in;
        in.depth = 1 + i % kDepth;
        auto vec = [&](double s) { return v3(uni(-s, s), uni(-s, s), uni(-s, s)); };
        auto unit = [](V3<double> v) { return v * (1.0 / length(v)); };
        in.S = vec(50.0);
        in.R = vec(50.0);
        for (int q = 0; q < in.depth; ++q) {
            in.n[q] = unit(vec(1.0));
            in.off[q] = uni(-80.0, 80.0);
            in.slab[q] = Slab<double>{uni(1.5, 9.0), std::pow(10.0, uni(-3.0, 0.5)), 1.0, uni(0.5, 1.0), uni(0.01, 0.5)};
        }
        in.tx_pol = unit(vec(1.0));
        in.rx_pol = unit(vec(1.0));
        if (i % 10 == 0) {  // normal incidence: every axis takes its fallback
            in.depth = 1;
            in.R = in.S + in.n[0] * 3.0;
            in.off[0] = dot(in.n[0], in.R) + 7.0;
        }
        in.f = std::pow(10.0, uni(8.7, 10.7));
        const double sq = 1.3, gg = uni(-1.0, 1.0), gr = uni(-1.0, 1.0), gi = uni(-1.0, 1.0);
        const Cx<DL> want = dual_reflection(in, sq);
        ReflectionRecordGrad<kDepth> g;
        const Cx<double> pf = reflection_record_vjp(in, sq, gg, gr, gi, g);
        double got[kLanes] = {g.S.x, g.S.y, g.S.z, g.R.x, g.R.y, g.R.z};
        int at = 6;
        for (int q = 0; q < in.depth; ++q)
            for (double v : {g.n[q].x, g.n[q].y, g.n[q].z, g.off[q], g.eps[q], g.sig[q]}) got[at++] = v;
        got[at++] = g.f;
        const double amp = std::hypot(want.re.v, want.im.v);
        refl = std::max(refl, worst(pf, want.re.v, want.im.v, amp + 1e-300));
        for (int l = 0; l < at; ++l) {
            const double re = want.re.d[l], im = want.im.d[l];
            const double ref = gg * 2.0 * (want.re.v * re + want.im.v * im) + gr * re + gi * im;
            const double scale = (2.0 * std::fabs(gg) * amp + std::fabs(gr) + std::fabs(gi)) * std::hypot(re, im);
            refl = std::max(refl, std::fabs(got[l] - ref) / (scale + 1e-300));
        }
    }
    std::printf("jets %.3g %.3g %.3g\n", term, face, refl);
    return 0;
}
"""


@pytest.fixture(scope="module")
def output(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("utd")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-D__noinline__=", f"-I{CUDA_INCLUDE}", f"-I{CSRC}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout.splitlines()


def _exact(x):
    """F(x) and (1+j)/2 - (C + jS)(x) from w(z) = e^{-z^2} erfc(-jz)."""
    w_of = lambda u: wofz(1j * np.exp(1j * np.pi / 4) * u)  # e^{j u^2} erfc(e^{j pi/4} u)
    F = 2j * np.sqrt(x) * 0.5 * np.sqrt(np.pi) * np.exp(-0.25j * np.pi) * w_of(np.sqrt(x))
    z = x * np.sqrt(np.pi / 2)
    c = np.exp(0.5j * np.pi * np.fmod(x * x, 4.0)) * np.conj(w_of(z)) * (1 + 1j) / 2
    return F, c


def test_transition_and_fresnel_complement(output):
    v = np.array([[float(t) for t in line.split()] for line in output[:-1]])
    x = v[:, 0]
    F, c = _exact(x)
    tol = np.where((x >= 400.0) & (x < 3e3), 8e-14, 4e-15) + 1e-13  # 1e-13: wofz
    assert np.all(np.abs(v[:, 1] + 1j * v[:, 2] - F) <= tol * np.abs(F))
    ok = x < 1e3  # x^2 beyond this leaves too few digits of the phase in the check itself
    rounding = 4e-16 * np.pi * x**2 + 1e-13
    assert np.all(np.abs(v[:, 3] + 1j * v[:, 4] - c)[ok] <= (rounding * np.abs(c))[ok])
    xf = x.astype(np.float32).astype(np.float64)
    F, c = _exact(xf)
    assert np.all(np.abs(v[:, 5] + 1j * v[:, 6] - F) <= 1e-6 * np.abs(F))
    assert np.all(np.abs(v[:, 7] + 1j * v[:, 8] - c)[ok] <= 1e-6 * np.abs(c)[ok])


def test_closed_form_jacobians_equal_dual_lanes(output):
    term, face, _ = (float(t) for t in output[-1].split()[1:])
    assert term <= 1e-9
    assert face <= 1e-9


def test_reflection_reverse_mode_equals_dual_lanes(output):
    assert float(output[-1].split()[3]) <= 1e-7
