// The error bound of the certified exact scan (csrc/cert_bound.h) against a
// model of the tensor cores' accumulation: groups of 4, 8 or 16 products and the
// accumulator, aligned to the largest and cut at 24 bits, the sum cut to a
// float.  The modelled distance, with the kernel's float32 epilogue, must lie
// within the bound of the reference's float32 distance.  Prints "ok <worst
// fraction of the bound>" or the first failure.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "cert_bound.h"

static float bf16(float v) {
    uint32_t u;
    std::memcpy(&u, &v, 4);
    u += 0x7fffu + ((u >> 16) & 1u);
    u &= 0xffff0000u;
    std::memcpy(&v, &u, 4);
    return v;
}

// v cut toward zero to a multiple of 2^(top - 23)
static double cut(double v, int top) { return std::ldexp(std::trunc(std::ldexp(v, 23 - top)), top - 23); }

static double mma(const std::vector<float>& q, const std::vector<float>& x, int group) {
    double acc = 0;
    const size_t n = (q.size() + 63) / 64 * 64;
    for (size_t b = 0; b < n; b += group) {
        double p[17], big = std::fabs(acc);
        for (int i = 0; i < group; i++) {
            p[i] = b + i < q.size() ? (double)q[b + i] * x[b + i] : 0.0;
            big = std::fmax(big, std::fabs(p[i]));
        }
        if (big == 0) continue;
        const int top = std::ilogb(big);
        double s = cut(acc, top);
        for (int i = 0; i < group; i++) s += cut(p[i], top);
        acc = s == 0 ? 0 : cut(s, std::ilogb(s));
    }
    return acc;
}

// the reference's distance: 16 accumulators, then the rest one by one
static float dist32(int space, const std::vector<float>& q, const std::vector<float>& x) {
    float a[16] = {0}, rest = 0;
    const size_t n16 = q.size() / 16 * 16;
    for (size_t i = 0; i < n16; i++) {
        const float t = space == 0 ? q[i] - x[i] : q[i];
        a[i % 16] = std::fma(t, space == 0 ? t : x[i], a[i % 16]);
    }
    float r = 0;
    for (float v : a) r += v;
    for (size_t i = n16; i < q.size(); i++) rest += space == 0 ? (q[i] - x[i]) * (q[i] - x[i]) : q[i] * x[i];
    r += rest;
    return space == 0 ? r : 1.0f - r;
}

static float square(const std::vector<float>& v) {
    float s = 0;
    for (float e : v) s = std::fma(e, e, s);
    return s;
}

static double worst = 0;

static bool check(const char* what, const std::vector<float>& q, const std::vector<float>& x) {
    std::vector<float> qb, xb, qe, xe;
    for (float v : q) {
        qb.push_back(bf16(v));
        qe.push_back(v - qb.back());
    }
    for (float v : x) {
        xb.push_back(bf16(v));
        xe.push_back(v - xb.back());
    }
    for (int space = 0; space < 2; space++)
        for (int group : {4, 8, 16}) {
            const float s = (float)mma(qb, xb, group);
            const double tc = space == 0 ? (double)std::fma(s, -2.0f, square(x)) + square(q) : 1.0 - (double)s;
            const double err = std::fabs(tc - dist32(space, q, x));
            const double bound =
                hnswgpu::cert_bound(space, (uint32_t)q.size(), std::sqrt((double)square(q)) * 1.001, std::sqrt((double)square(qe)) * 1.001,
                                    std::sqrt((double)square(x)) * 1.001, std::sqrt((double)square(xe)) * 1.001);
            worst = std::fmax(worst, err / bound);
            if (!(err <= bound)) {
                std::printf("%s, dim %zu, space %d, groups of %d: error %g, bound %g\n", what, q.size(), space, group, err, bound);
                return false;
            }
        }
    return true;
}

int main() {
    std::mt19937 rng(7);
    std::normal_distribution<float> normal;
    for (size_t dim : {1, 3, 16, 17, 33, 64, 100, 128, 200, 768, 1000, 2048, 2800})
        for (int t = 0; t < 12; t++) {
            std::vector<float> q(dim), x(dim);
            for (size_t i = 0; i < dim; i++) q[i] = normal(rng), x[i] = normal(rng);
            if (!check("normal", q, x)) return 1;
            for (size_t i = 0; i < dim; i++) x[i] = q[i] + 0.01f * normal(rng);
            if (!check("close", q, x)) return 1;
            for (size_t i = 0; i < dim; i++) q[i] = (float)(rng() % 256), x[i] = (float)(rng() % 256);
            if (!check("bytes", q, x)) return 1;
            for (size_t i = 0; i < dim; i++) x[i] = std::fmin(255.f, q[i] + (float)(rng() % 3));
            if (!check("close bytes", q, x)) return 1;
            // one large product, and every later one just under the last bit kept of it
            for (size_t i = 0; i < dim; i++) q[i] = std::ldexp(1.f, -11), x[i] = std::ldexp(1.9921875f, -13);
            q[0] = x[0] = 1;
            if (!check("one large product", q, x)) return 1;
            for (size_t i = 1; i < dim; i++)
                if (rng() % 2) x[i] = -x[i];
            if (!check("one large product, both signs", q, x)) return 1;
        }
    std::printf("ok %.3f\n", worst);
    return 0;
}
