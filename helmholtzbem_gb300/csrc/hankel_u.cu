// The table of hankel_u.cuh, made on the device in double-double arithmetic
// (Dekker 1971 / Knuth: an unevaluated sum of two doubles, about 106 bits).
#include <mutex>

#include "hankel_u.cuh"

namespace hbem {

namespace {

struct dd {
    double h, l;
};

#define HD __host__ __device__ inline

HD dd mkd(double h, double l = 0.) { dd z; z.h = h; z.l = l; return z; }
HD dd quick(double a, double b) { const double s = a + b; return mkd(s, b - (s - a)); }
HD dd two_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return mkd(s, (a - (s - t)) + (b - t));
}
HD dd operator+(dd a, dd b) {
    dd s = two_sum(a.h, b.h);
    const dd t = two_sum(a.l, b.l);
    s = quick(s.h, s.l + t.h);
    return quick(s.h, s.l + t.l);
}
HD dd operator-(dd a) { return mkd(-a.h, -a.l); }
HD dd operator-(dd a, dd b) { return a + (-b); }
HD dd operator*(dd a, dd b) {
    const double p = a.h * b.h;
    return quick(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
HD dd operator*(double a, dd b) { return mkd(a) * b; }
HD dd operator/(dd a, dd b) {
    const double q1 = a.h / b.h;
    dd r = a - q1 * b;
    const double q2 = r.h / b.h;
    r = r - q2 * b;
    return quick(q1, q2) + mkd(r.h / b.h);
}
HD dd operator/(dd a, double b) { return a / mkd(b); }
HD dd dsqrt(dd a) {
    const double x = sqrt(a.h);
    const dd r = a - mkd(x) * mkd(x);
    const dd y = mkd(x) + mkd(r.h / (2. * x));
    return y + (a - y * y) / (2. * x);          // one more Newton step
}

HD dd dd_ln2() { return mkd(0.6931471805599453, 2.319046813846299e-17); }
HD dd dd_gamma() { return mkd(0.5772156649015329, -4.942915152430645e-18); }
HD dd dd_pi() { return mkd(3.141592653589793, 1.2246467991473532e-16); }

HD dd dexp(dd a) {
    const double k = rint(a.h / 0.6931471805599453);
    const dd r = (a - k * dd_ln2()) / 512.;
    dd t = mkd(1.), s = mkd(1.);
    for (int m = 1; m <= 12; ++m) {
        t = t * r / (double)m;
        s = s + t;
    }
    for (int q = 0; q < 9; ++q) s = s * s;
    const double sc = ldexp(1., (int)k);
    return mkd(s.h * sc, s.l * sc);
}
HD dd dlog(dd a) {
    const double y = log(a.h);
    const dd r = a * dexp(mkd(-y)) - mkd(1.);
    return mkd(y) + (r - 0.5 * (r * r));
}
HD void dsincos(dd x, dd& s, dd& c) {
    const double n = rint(x.h * 0.6366197723675814);
    dd r = x - n * mkd(1.5707963267948966, 6.123233995736766e-17);
    r = r + mkd(n * 1.4973849048591833e-33);   // third part of -pi/2
    const dd r2 = r * r;
    dd t = r, ss = r, u = mkd(1.), cc = mkd(1.);
    for (int m = 1; m <= 14; ++m) {
        u = -(u * r2) / (double)((2 * m - 1) * (2 * m));
        cc = cc + u;
        t = -(t * r2) / (double)((2 * m) * (2 * m + 1));
        ss = ss + t;
    }
    const int q = (int)((long long)n & 3);
    if (q == 0) { s = ss; c = cc; }
    else if (q == 1) { s = cc; c = -ss; }
    else if (q == 2) { s = -ss; c = -cc; }
    else { s = -cc; c = ss; }
}

// J_m(x) / x^m and Y_m(x) / x^m, m = 0..7, at u = x^2
HD void scaled_bessel(double u, dd* j, dd* y) {
    const dd U = mkd(u);
    if (u <= 625.) {
        const dd w = mkd(-0.25 * u);
        // ascending series (DLMF 10.2.2, 10.8.1)
        dd lead = mkd(1.);                       // 1 / (2^m m!)
        for (int m = 0; m < 8; ++m) {
            if (m) lead = lead / (2. * m);
            dd t = lead, s = lead;
            for (int k = 1; k < 90; ++k) {
                t = t * w / (double)(k * (m + k));
                s = s + t;
                if (fabs(t.h) < 1e-34 * lead.h) break;
            }
            j[m] = s;
        }
        const dd L = 0.5 * dlog(-w) + dd_gamma(), ip = mkd(1.) / dd_pi();
        dd t = mkd(1.), H = mkd(0.), s0 = mkd(0.), t1 = mkd(1.), s1 = mkd(1.);   // k = 0: H_0 + H_1 = 1
        for (int k = 1; k < 90; ++k) {
            H = H + mkd(1.) / (double)k;
            t = t * w / (double)((long long)k * k);
            s0 = s0 - H * t;
            t1 = t1 * w / (double)((long long)k * (k + 1));
            s1 = s1 + (H + H + mkd(1.) / (double)(k + 1)) * t1;
            if (fabs(t.h) < 1e-36) break;
        }
        y[0] = (2. * ip) * (L * j[0] + s0);
        y[1] = (2. * ip) * (L * j[1]) - (0.5 * ip) * s1 - (2. * ip) / U;
    } else {
        // Hankel's expansion (DLMF 10.17.5)
        const dd x = dsqrt(U);
        dd s, c;
        dsincos(x, s, c);
        const dd a = s + c, b = s - c, sc = mkd(1.) / dsqrt(dd_pi() * x);
        for (int nu = 0; nu < 2; ++nu) {
            dd t = mkd(1.), P = mkd(1.), Q = mkd(0.);
            double last = 1.;
            for (int k = 1; k < 60; ++k) {
                t = (double)(4 * nu - (2 * k - 1) * (2 * k - 1)) * t / ((8. * k) * x);
                if (fabs(t.h) > last) break;
                last = fabs(t.h);
                // i^k t_k: +i, -1, -i, +1
                if (k & 1) Q = (k & 2) ? Q - t : Q + t;
                else P = (k & 2) ? P - t : P + t;
                if (last < 1e-33) break;
            }
            if (nu == 0) {
                j[0] = sc * (P * a - Q * b);
                y[0] = sc * (P * b + Q * a);
            } else {
                j[1] = sc * (P * b + Q * a) / x;
                y[1] = sc * (Q * b - P * a) / x;
            }
        }
        for (int m = 1; m < 7; ++m) j[m + 1] = ((2. * m) * j[m] - j[m - 1]) / U;
    }
    for (int m = 1; m < 7; ++m) y[m + 1] = ((2. * m) * y[m] - y[m - 1]) / U;
}

HD void make_entry(int idx, HkEntry* out) {
    int e = kHkEMin;
    while (e + 1 < kHkEMax && hk_base(e + 1) <= idx) ++e;
    const int b = hk_bits(e);
    const double hw = ldexp(1., e - b - 1);
    const double u = ldexp(1., e) + (2 * (idx - hk_base(e)) + 1) * hw;
    dd j[8], y[8];
    scaled_bessel(u, j, y);
    double fac = 1.;          // (-1/2)^m / m!, exact to rounding: applied in double-double
    dd F = mkd(1.);
    dd jr[8], yr[8];
    for (int m = 0; m < 8; ++m) {
        if (m) F = F / (-2. * m);
        jr[m] = F * j[m];
        yr[m] = F * y[m];
    }
    for (int m = 0; m < 7; ++m, fac *= hw) {
        const dd gj = (-2. * (m + 1)) * jr[m + 1], gy = (-2. * (m + 1)) * yr[m + 1];
        const double v[2][2] = {{jr[m].h * fac, yr[m].h * fac}, {gj.h * fac, gy.h * fac}};
        for (int q = 0; q < 2; ++q)
            for (int r = 0; r < 2; ++r) {
                if (m < 4) out->c[q][m][r] = v[q][r];
                else out->s[q][m - 4][r] = (float)v[q][r];
            }
    }
}

__global__ void __launch_bounds__(64) k_hankel_table(HkEntry* tab) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < kHkEntries) make_entry(idx, tab + idx);
}

__device__ HkEntry g_hk_table[kHkEntries];

std::mutex g_hk_mu;
bool g_hk_made[64];

}  // namespace

const HkEntry* hankel_table(cudaError_t* err) {
    int dev = 0;
    *err = cudaGetDevice(&dev);
    if (*err != cudaSuccess) return nullptr;
    if (dev < 0 || dev >= 64) {
        *err = cudaErrorInvalidDevice;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(g_hk_mu);
    void* p = nullptr;   // asked for each time: a device reset may move the array
    *err = cudaGetSymbolAddress(&p, g_hk_table);
    if (*err != cudaSuccess) return nullptr;
    if (g_hk_made[dev]) {   // a device reset in between clears it (its entries are never zero)
        double first = 0.;
        *err = cudaMemcpy(&first, p, sizeof(double), cudaMemcpyDeviceToHost);
        if (*err != cudaSuccess) return nullptr;
        if (first != 0.) return static_cast<const HkEntry*>(p);
        g_hk_made[dev] = false;
    }
    k_hankel_table<<<(kHkEntries + 63) / 64, 64>>>(static_cast<HkEntry*>(p));
    *err = cudaGetLastError();
    if (*err == cudaSuccess) *err = cudaStreamSynchronize(0);   // complete before any stream reads it
    if (*err != cudaSuccess) return nullptr;
    g_hk_made[dev] = true;
    return static_cast<const HkEntry*>(p);
}

}  // namespace hbem
