// Reverse mode of one reflection record's path field: one FP64 forward sweep
// (images, hits, the Jones chain) that keeps each bounce's incoming field, then
// one reverse sweep that returns the gradient with respect to every input at
// once.  A dual-number evaluation repeats the whole chain once per four
// parameters (up to 13 passes with vertices) and spills its lanes.
//
// Every branch (normalisation fallbacks, the orientation of the normal, the
// clamps of the Fresnel laws) is differentiated on the side the forward value
// took, as the dual evaluation does.  Adjoint conventions: utd_adjoint.cuh.
#pragma once

#include "em.cuh"
#include "utd_adjoint.cuh"

namespace wcb {

namespace rev {

// y = safe_normalize(v, fallback)
WCB_HD void safe_normalize_vjp(D3 v, D3 fallback, D3 yb, D3& vb, D3& fb) {
    const double n = length(v);
    if (n > kUtdSmallEps) {
        const double inv = 1.0 / (n + kUtdEps);
        vb = vb + yb * inv - v * (dot(yb, v) * inv * inv / n);
        return;
    }
    const double fn = length(fallback);
    const double inv = 1.0 / (fn + kUtdEps);
    fb = fb + yb * inv;
    if (fn > 0.0) fb = fb - fallback * (dot(yb, fallback) * inv * inv / fn);
}

// y = transverse(dir, p) = p - dir (p . dir); p's adjoint is added to pb
WCB_HD void transverse_vjp(D3 dir, D3 p, D3 yb, D3& dirb, D3& pb) {
    const double yd = dot(yb, dir);
    dirb = dirb - yb * dot(p, dir) - p * yd;
    pb = pb + yb - dir * yd;
}

// y = safe_normalize(a x b, stable_perp_basis(dir, pref)) with its fallback's
// own normalisation; the fallback is only differentiated where it is taken.
WCB_HD void axis_vjp(D3 a, D3 b, D3 dir, D3 pref, D3 yb, D3& ab, D3& bb, D3& dirb, D3& prefb) {
    const D3 v = cross(a, b);
    if (length(v) > kUtdSmallEps) {
        D3 vb = zero3(), none = zero3();
        safe_normalize_vjp(v, v, yb, vb, none);
        cross_vjp(a, b, vb, ab, bb);
        return;
    }
    const D3 alt = fabs(dir.z) < 0.9 ? v3(0.0, 0.0, 1.0) : v3(0.0, 1.0, 0.0);
    const D3 proj = transverse(dir, pref), alt_proj = transverse(dir, alt);
    const D3 perp = safe_normalize(proj, alt_proj);
    D3 perpb = zero3(), none = zero3(), projb = zero3(), altb = zero3();
    safe_normalize_vjp(v, perp, yb, none, perpb);
    safe_normalize_vjp(proj, alt_proj, perpb, projb, altb);
    transverse_vjp(dir, pref, projb, dirb, prefb);
    none = zero3();
    transverse_vjp(dir, alt, altb, dirb, none);
}

}  // namespace rev

// Thin-slab Fresnel coefficients (slab_fresnel, wavelength c / f) with their
// derivatives by cos, eps_r, sigma_e and frequency.
WCB_HD void slab_jet(double cos_theta, const Slab<double>& m, double f, FaceJet& out) {
    const double omega = s_max(kTwoPi * f, kUtdSmallEps);
    const double raw = fabs(cos_theta);
    const bool ct_in = raw >= kUtdSmallEps && raw <= 1.0;
    const double ct = fmin(fmax(raw, kUtdSmallEps), 1.0);
    const double dct = ct_in ? (cos_theta < 0.0 ? -1.0 : 1.0) : 0.0;
    const bool eps_in = m.eps_r >= kUtdSmallEps, sig_in = m.sigma_e >= 0.0;
    const double loss = (sig_in ? m.sigma_e : 0.0) / (omega * kEps0);
    const Cx<double> eta = cx(eps_in ? m.eps_r : kUtdSmallEps, -loss);
    const double mu = fmax(m.mu_r, kUtdSmallEps);
    const Cx<double> root = csqrt(eta * mu - cx(fmax(1.0 - ct * ct, 0.0), 0.0));
    const Cx<double> one = cx(1.0, 0.0);
    const Cx<double> a = cx(mu * ct, 0.0), b = eta * ct;
    const Cx<double> ia = one / (a + root), ib = one / (b + root);
    const Cx<double> te = (a - root) * ia, tm = (b - root) * ib;
    const double wavelength = kC0 / f;
    const bool wl_in = wavelength >= kUtdSmallEps;
    const double scale = kTwoPi * fmax(m.thickness, 0.0) / (wl_in ? wavelength : kUtdSmallEps);
    const Cx<double> q = root * scale;
    const Cx<double> phase = cexp(cx(2.0 * q.im, -2.0 * q.re));
    const Cx<double> te2 = te * te, tm2 = tm * tm;
    const Cx<double> de = one / (one - te2 * phase), dm = one / (one - tm2 * phase);
    const Cx<double> open = one - phase;
    out.te = te * open * de * m.gain;
    out.tm = tm * open * dm * m.gain;
    // r = g i (1 - P) / (1 - i^2 P): dr/di = g (1 - P)(1 + i^2 P) / den^2, dr/dP = g i (i^2 - 1) / den^2
    const Cx<double> ge = de * de * m.gain, gm = dm * dm * m.gain;
    const Cx<double> te_i = open * (one + te2 * phase) * ge, te_p = te * (te2 - one) * ge;
    const Cx<double> tm_i = open * (one + tm2 * phase) * gm, tm_p = tm * (tm2 - one) * gm;
    const Cx<double> inv_root = one / root;
    const Cx<double> qa = ia * ia * 2.0, qb = ib * ib * 2.0;
    const Cx<double> m2jp = cx(2.0 * phase.im, -2.0 * phase.re);  // -2j P
    auto lane = [&](int l, double dc, Cx<double> deta, double dscale) {
        const Cx<double> ds = (deta * mu + cx(2.0 * ct * dc, 0.0)) * inv_root * 0.5;
        const Cx<double> dte = (root * (mu * dc) - a * ds) * qa;
        const Cx<double> dtm = (root * (deta * ct + eta * dc) - b * ds) * qb;
        const Cx<double> dp = m2jp * (ds * scale + root * dscale);
        out.dte[l] = te_i * dte + te_p * dp;
        out.dtm[l] = tm_i * dtm + tm_p * dp;
    };
    const Cx<double> none = cx(0.0, 0.0);
    lane(0, dct, none, 0.0);
    lane(1, 0.0, cx(eps_in ? 1.0 : 0.0, 0.0), 0.0);
    lane(2, 0.0, cx(0.0, sig_in ? -1.0 / (omega * kEps0) : 0.0), 0.0);
    lane(3, 0.0, cx(0.0, kTwoPi * f >= kUtdSmallEps ? loss * kTwoPi / omega : 0.0), wl_in ? scale / f : 0.0);
}

// Inputs of one reflection record's receiver coefficient and the gradient of
// the loss with respect to them (plane q: unit normal n, offset off).
template <int D>
struct ReflectionRecordIn {
    V3<double> S, R, tx_pol, rx_pol;
    int depth;
    V3<double> n[D];
    double off[D];
    Slab<double> slab[D];
    double f;
};
template <int D>
struct ReflectionRecordGrad {
    V3<double> S, R, n[D];
    double off[D], eps[D], sig[D], f;
};

// The record's path field sq * coefficient and, for the loss
// gg |pf|^2 + gr Re(pf) + gi Im(pf) around it, the gradient by every input.
template <int D>
WCB_HD Cx<double> reflection_record_vjp(const ReflectionRecordIn<D>& in, double sq, double gg, double gr, double gi,
                                        ReflectionRecordGrad<D>& g) {
    using rev::D3;
    using rev::rdot;
    using rev::zero3;
    const int d = in.depth;
    const double k = in.f * (kTwoPi / kC0);
    const D3 ez = v3(0.0, 0.0, 1.0);
    // ------------------------------------------------------------ forward sweep
    D3 img[D], hit[D];
    D3 p = in.S;
    for (int q = 0; q < d; ++q) {
        p = p - in.n[q] * (2.0 * (dot(p, in.n[q]) - in.off[q]));
        img[q] = p;
    }
    D3 x = in.R;
    for (int q = d - 1; q >= 0; --q) {
        const D3 e = img[q] - x;
        x = x + e * ((in.off[q] - dot(x, in.n[q])) / dot(e, in.n[q]));
        hit[q] = x;
    }
    const D3 unfolded = in.R - p;
    const double Lr = length(unfolded);
    const bool L_in = Lr >= kUtdEps;
    const double L = L_in ? Lr : kUtdEps;
    C3<double> value[D + 1];  // the field before each bounce
    D3 out[D + 1];            // the direction before each bounce (fallback of its incident direction)
    out[0] = safe_normalize(hit[0] - in.S, ez);
    value[0] = c3_from_real(transverse(out[0], in.tx_pol));
    FaceJet jet;
    D3 inc, nn, refl, s_axis, p_in, p_out;
    auto bounce = [&](int q) {
        inc = safe_normalize(hit[q] - (q > 0 ? hit[q - 1] : in.S), out[q]);
        nn = safe_normalize(in.n[q], ez);
        if (dot(inc, nn) > 0.0) nn = -nn;
        const double di = dot(inc, nn);
        refl = safe_normalize(inc - nn * (2.0 * di), -inc);
        s_axis = safe_normalize(cross(nn, inc), stable_perp_basis(inc, nn));
        p_in = safe_normalize(cross(s_axis, inc), stable_perp_basis(inc, s_axis));
        p_out = safe_normalize(cross(s_axis, refl), stable_perp_basis(refl, s_axis));
        slab_jet(fabs(di), in.slab[q], in.f, jet);
    };
#pragma unroll 1
    for (int q = 0; q < d; ++q) {
        bounce(q);
        value[q + 1] = c3_axis(s_axis, jet.te * c3_dot(value[q], s_axis)) +
                       c3_axis(p_out, jet.tm * c3_dot(value[q], p_in));
        out[q + 1] = refl;
    }
    const D3 leg = in.R - hit[d - 1];
    const D3 dir = safe_normalize(leg, out[d]);
    const D3 rxt = transverse(dir, in.rx_pol);
    const Cx<double> c0 = c3_dot(value[d], rxt);
    const double amp = 1.0 / (2.0 * k * L);
    const Cx<double> carrier = phasor_neg_kd<double>(k, Lr) * amp;
    const Cx<double> coef = carrier * c0;
    const Cx<double> pf = coef * sq;

    // ------------------------------------------------------------ reverse sweep
    const Cx<double> coefb = cx(2.0 * gg * pf.re + gr, 2.0 * gg * pf.im + gi) * sq;
    const Cx<double> carrierb = coefb * cconj(c0), c0b = coefb * cconj(carrier);
    const Cx<double> mj = cx(carrier.im, -carrier.re);  // -j carrier
    const double Lb = rdot(carrierb, mj) * k - (L_in ? rdot(carrierb, carrier) / L : 0.0);
    const double kb = rdot(carrierb, mj) * Lr - rdot(carrierb, carrier) / k;
    g.f = kb * (kTwoPi / kC0);
    C3<double> vb{c0b * rxt.x, c0b * rxt.y, c0b * rxt.z};
    D3 dirb = zero3(), none = zero3(), legb = zero3(), outb = zero3(), Rb = zero3(), Sb = zero3();
    rev::transverse_vjp(dir, in.rx_pol, v3(rdot(c0b, value[d].x), rdot(c0b, value[d].y), rdot(c0b, value[d].z)), dirb,
                        none);
    rev::safe_normalize_vjp(leg, out[d], dirb, legb, outb);
    Rb = Rb + legb;
    D3 hitb[D];
    for (int q = 0; q < d; ++q) hitb[q] = zero3();
    hitb[d - 1] = hitb[d - 1] - legb;
#pragma unroll 1
    for (int q = d - 1; q >= 0; --q) {
        bounce(q);
        const C3<double>& v = value[q];
        const Cx<double> es = c3_dot(v, s_axis), ep = c3_dot(v, p_in);
        const Cx<double> A = jet.te * es, B = jet.tm * ep;
        const Cx<double> Ab = c3_dot(vb, s_axis), Bb = c3_dot(vb, p_out);
        D3 sb = v3(rdot(vb.x, A), rdot(vb.y, A), rdot(vb.z, A));
        const D3 pob = v3(rdot(vb.x, B), rdot(vb.y, B), rdot(vb.z, B));
        const Cx<double> teb = Ab * cconj(es), esb = Ab * cconj(jet.te);
        const Cx<double> tmb = Bb * cconj(ep), epb = Bb * cconj(jet.tm);
        vb = c3_axis(s_axis, esb) + c3_axis(p_in, epb);
        sb = sb + v3(rdot(esb, v.x), rdot(esb, v.y), rdot(esb, v.z));
        const D3 pib = v3(rdot(epb, v.x), rdot(epb, v.y), rdot(epb, v.z));
        double lanes[4];
        for (int l = 0; l < 4; ++l) lanes[l] = rdot(teb, jet.dte[l]) + rdot(tmb, jet.dtm[l]);
        g.eps[q] = lanes[1];
        g.sig[q] = lanes[2];
        g.f += lanes[3];
        const double di = dot(inc, nn);
        double dib = di < 0.0 ? -lanes[0] : lanes[0];
        D3 reflb = outb, incb = zero3(), nnb = zero3();
        rev::axis_vjp(s_axis, refl, refl, s_axis, pob, sb, reflb, reflb, sb);
        rev::axis_vjp(s_axis, inc, inc, s_axis, pib, sb, incb, incb, sb);
        rev::axis_vjp(nn, inc, inc, nn, sb, nnb, incb, incb, nnb);
        // refl = safe_normalize(inc - 2 nn (inc . nn), -inc)
        D3 rawb = zero3(), negb = zero3();
        rev::safe_normalize_vjp(inc - nn * (2.0 * di), -inc, reflb, rawb, negb);
        incb = incb + rawb - negb;
        dib -= 2.0 * dot(rawb, nn);
        nnb = nnb - rawb * (2.0 * di);
        incb = incb + nn * dib;
        nnb = nnb + inc * dib;
        // the oriented unit normal
        D3 nb = zero3();
        none = zero3();
        const bool flipped = dot(nn, safe_normalize(in.n[q], ez)) < 0.0;
        rev::safe_normalize_vjp(in.n[q], ez, flipped ? -nnb : nnb, nb, none);
        g.n[q] = nb;
        // the incident direction
        D3 segb = zero3();
        outb = zero3();
        const D3 prev = q > 0 ? hit[q - 1] : in.S;
        rev::safe_normalize_vjp(hit[q] - prev, out[q], incb, segb, outb);
        hitb[q] = hitb[q] + segb;
        if (q > 0) hitb[q - 1] = hitb[q - 1] - segb;
        else Sb = Sb - segb;
    }
    // the launch direction and polarisation
    none = zero3();
    rev::transverse_vjp(out[0], in.tx_pol, v3(vb.x.re, vb.y.re, vb.z.re), outb, none);
    D3 launchb = zero3();
    none = zero3();
    rev::safe_normalize_vjp(hit[0] - in.S, ez, outb, launchb, none);
    hitb[0] = hitb[0] + launchb;
    Sb = Sb - launchb;
    // hits, from the first bounce up: x_out = x + e t, t = (off - x.n) / (e.n), e = img - x
    D3 imgb[D];
    for (int q = 0; q < d; ++q) {
        const D3 xi = q + 1 < d ? hit[q + 1] : in.R;
        const D3 e = img[q] - xi;
        const double den = dot(e, in.n[q]);
        const double t = (in.off[q] - dot(xi, in.n[q])) / den;
        const D3 xb = hitb[q];
        const double tb = dot(xb, e);
        const double numb = tb / den, denb = -tb * t / den;
        const D3 eb = xb * t + in.n[q] * denb;
        g.n[q] = g.n[q] + e * denb - xi * numb;
        g.off[q] = numb;
        imgb[q] = eb;
        const D3 xib = xb - in.n[q] * numb - eb;
        if (q + 1 < d) hitb[q + 1] = hitb[q + 1] + xib;
        else Rb = Rb + xib;
    }
    if (Lr > 0.0) {
        const D3 ub = unfolded * (Lb / Lr);
        Rb = Rb + ub;
        imgb[d - 1] = imgb[d - 1] - ub;
    }
    // images: p_out = p - 2 n h, h = p.n - off
    D3 pb = zero3();
    for (int q = d - 1; q >= 0; --q) {
        pb = pb + imgb[q];
        const D3 pin = q > 0 ? img[q - 1] : in.S;
        const double h = dot(pin, in.n[q]) - in.off[q];
        const double hb = -2.0 * dot(pb, in.n[q]);
        g.n[q] = g.n[q] - pb * (2.0 * h) + pin * hb;
        g.off[q] -= hb;
        pb = pb + in.n[q] * hb;
    }
    g.S = Sb + pb;
    g.R = Rb;
    return pf;
}

}  // namespace wcb
