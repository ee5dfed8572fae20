// The collision compiled for the host, in FP32 and FP64, on [27][n] populations.
#include <cmath>
using std::fabs;
using std::fma;

#include "../../lbm3_b200/csrc/cumulant.cuh"

namespace {
template <class T> void collide(T* f, int n, T nu, T limiter) {
    const auto P = lbm::makeCollisionConstsT<T>(nu, T(1), limiter);
    for (int c = 0; c < n; ++c) {
        T v[27];
        for (int d = 0; d < 27; ++d) v[d] = f[d * n + c];
        lbm::collideCumulantT<T>(v, P, P.lambda, T(0), T(0), T(0));
        for (int d = 0; d < 27; ++d) f[d * n + c] = v[d];
    }
}
}  // namespace

extern "C" void collide_check_f32(float* f, int n, float nu, float limiter) { collide<float>(f, n, nu, limiter); }
extern "C" void collide_check_f64(double* f, int n, double nu, double limiter) { collide<double>(f, n, nu, limiter); }
