// The device rules that tests check on the CPU: the shading and triangle headers compiled for the host, where
// arithmetic rounds as on the device (no contraction), behind a few array functions.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __noinline__
#define __noinline__ __attribute__((noinline))
#endif

using std::isfinite;
using std::isnan;

namespace {
template <class To, class From>
To bits_as(From v) {
    To out;
    std::memcpy(&out, &v, sizeof(out));
    return out;
}
inline float __int_as_float(int v) { return bits_as<float>(v); }
inline int __float_as_int(float v) { return bits_as<int>(v); }
inline float __double2float_rn(double v) { return static_cast<float>(v); }
inline uint32_t __float_as_uint(float v) { return bits_as<uint32_t>(v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
}  // namespace

#include "bf200_shading.cuh"
#include "bf200_triangle.cuh"

using namespace bf200;

namespace {
// n products of NN columns over ND columns: the direct form, whether it applies, and both split forms.
template <int NN, int ND>
void products(const float* num, const float* den, uint64_t n, float* direct, uint8_t* applies, float* quotient,
              float* ratio) {
    for (uint64_t i = 0; i < n; ++i) {
        float a[NN], b[ND];
        for (int k = 0; k < NN; ++k) {
            a[k] = num[k * n + i];
        }
        for (int k = 0; k < ND; ++k) {
            b[k] = den[k * n + i];
        }
        const Factors<NN, ND> f(a, b);
        Lane lane;
        applies[i] = f.direct(direct[i]) ? 1 : 0;
        quotient[i] = factors_quotient(f, lane);
        ratio[i] = factors_ratio(f, lane);
    }
}
}  // namespace

extern "C" {

int rule_products(int nn, int nd, const float* num, const float* den, uint64_t n, float* direct, uint8_t* applies,
                  float* quotient, float* ratio) {
#define CASE(NN, ND)                                                            \
    if (nn == NN && nd == ND) {                                                 \
        products<NN, ND>(num, den, n, direct, applies, quotient, ratio);        \
        return 0;                                                               \
    }
    CASE(2, 1) CASE(3, 1) CASE(4, 1) CASE(2, 2) CASE(4, 3) CASE(5, 2) CASE(7, 2) CASE(7, 4)
#undef CASE
    return 1;
}

// positive_product2 and mis_weight beside their split forms (the weight's smaller density over its larger one)
void rule_product2(const float* a, const float* b, uint64_t n, float* out, float* split) {
    for (uint64_t i = 0; i < n; ++i) {
        Lane lane;
        out[i] = positive_product2(a[i], b[i], lane);
        split[i] = split_product2(a[i], b[i], lane);
    }
}

void rule_mis_weight(uint32_t heuristic, const float* sampled, const float* competing, uint64_t n, float* out) {
    for (uint64_t i = 0; i < n; ++i) {
        Lane lane;
        out[i] = mis_weight(heuristic, sampled[i], competing[i], lane);
    }
}

void rule_split_mis_ratio(uint32_t heuristic, const float* less, const float* more, uint64_t n, float* out) {
    for (uint64_t i = 0; i < n; ++i) {
        out[i] = split_mis_ratio(heuristic, less[i], more[i]);
    }
}

void rule_next_float(const float* v, uint32_t up, uint64_t n, float* out) {
    for (uint64_t i = 0; i < n; ++i) {
        out[i] = next_float(v[i], up != 0U);
    }
}

// certain_miss of rays against triangles, and the whole test: 0 miss, 1 hit, 2 failure, with (t, barycentrics)
void rule_triangles(const float* vertices, const float* origin, const float* direction, uint64_t n, uint8_t* certain,
                    uint8_t* code, float* out) {
    for (uint64_t i = 0; i < n; ++i) {
        const float* p = vertices + 9 * i;
        const float4 v0 = make_float4(p[0], p[1], p[2], 0.0F), v1 = make_float4(p[3], p[4], p[5], 0.0F),
                     v2 = make_float4(p[6], p[7], p[8], 0.0F);
        const F3 o{origin[3 * i], origin[3 * i + 1], origin[3 * i + 2]};
        const F3 d{direction[3 * i], direction[3 * i + 1], direction[3 * i + 2]};
        const float d_sum = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
        certain[i] = certain_miss(v0, v1, v2, o, d, d_sum) ? 1 : 0;
        TriangleHit hit{};
        code[i] = static_cast<uint8_t>(triangle_test(v0, v1, v2, o, d, 0.0F, kInf, true, hit));
        out[4 * i] = hit.t;
        out[4 * i + 1] = hit.b0;
        out[4 * i + 2] = hit.b1;
        out[4 * i + 3] = hit.b2;
    }
}
}
