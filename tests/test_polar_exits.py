"""The polar iteration's identity exits on badly conditioned deformation gradients (CPU).

polar_rotation (pk_math.cuh) leaves most of the reference's exit tests
(FEMModel::ExtractRotationPolar, FEMModel.cpp:115-163: the identity where an iterate's inverse
is not finite or its determinant is at most 1e-8) out of its common path.  Compiled for the
host without contraction, it must give the bits, the iterations and the fallback of the plain
iteration with every test, over deformation gradients whose singular values span up to twelve
decades.
"""
import os
import subprocess

import pytest

from physik_b200 import _lib as L

SOURCE = r"""
#include "pk_math.cuh"
#include <cstdio>
#include <cstring>
#include <random>
using namespace pk;
template <class T>
M3<T> plain(const M3<T>& f, int* its, bool* fallback)
{
    const T limit = T(1.0e-8);
    *its = 0;
    *fallback = true;
    if (!finite9(f) || fabs(det(f)) <= limit) return mident<T>();
    M3<T> r = f;
    for (int it = 0; it < 12; ++it) {
        *its = it + 1;
        const M3<T> ti = inverse(transpose(r));
        if (!finite9(ti) || fabs(det(ti)) <= limit) return mident<T>();
        const M3<T> next = scale(add(r, ti), T(0.5));
        if (!finite9(next)) return mident<T>();
        T diff = T(0);
        for (int c = 0; c < 3; ++c) {
            const V3<T> d = next.c[c] - r.c[c];
            diff += dot(d, d);
        }
        r = next;
        if (diff <= T(1.0e-10)) break;
    }
    if (!finite9(r)) return mident<T>();
    *fallback = false;
    if (det(r) < T(0)) r.c[2] = r.c[2] * T(-1);
    return r;
}
template <class T>
long differing(double span, long count, unsigned seed)
{
    std::mt19937_64 g(seed);
    std::normal_distribution<double> normal;
    std::uniform_real_distribution<double> log_size(-std::log(span), std::log(span));
    long bad = 0;
    for (long i = 0; i < count; ++i) {
        double q[2][3][3];
        for (auto& m : q)
            for (int k = 0; k < 3; ++k) {
                for (double& x : m[k]) x = normal(g);
                for (int j = 0; j < k; ++j) {
                    const double d = m[k][0] * m[j][0] + m[k][1] * m[j][1] + m[k][2] * m[j][2];
                    for (int e = 0; e < 3; ++e) m[k][e] -= d * m[j][e];
                }
                const double s = std::sqrt(m[k][0] * m[k][0] + m[k][1] * m[k][1] + m[k][2] * m[k][2]);
                for (double& x : m[k]) x /= s;
            }
        double s[3], v[3];
        for (double& x : s) x = std::exp(log_size(g));
        M3<T> f;
        for (int c = 0; c < 3; ++c) {
            for (int e = 0; e < 3; ++e) {
                v[e] = 0;
                for (int k = 0; k < 3; ++k) v[e] += q[0][k][e] * s[k] * q[1][k][c];
            }
            f.c[c] = V3<T>{T(v[0]), T(v[1]), T(v[2])};
        }
        int ia, ib;
        bool fa, fb;
        const M3<T> a = plain(f, &ia, &fa), b = polar_rotation<T>(f, &ib, &fb);
        bad += ia != ib || fa != fb || std::memcmp(&a, &b, sizeof a) != 0;
    }
    return bad;
}
int main()
{
    for (double span : {3.0, 1e2, 1e3, 1e4, 1e5, 1e6})
        std::printf("%g %ld %ld\n", span, differing<float>(span, 100000, 1), differing<double>(span, 50000, 2));
}
"""


def test_exits_are_those_of_the_plain_iteration(tmp_path):
    source, program = tmp_path / "polar.cpp", tmp_path / "polar"
    source.write_text(SOURCE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    kernels = os.path.join(L.ROOT, "physik_b200", "csrc", "kernels")
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", kernels, "-I",
                    os.path.join(cuda, "include"), str(source), "-o", str(program)], check=True)
    out = subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split()
    counts = [int(c) for i, c in enumerate(out) if i % 3]
    assert len(counts) == 12 and not any(counts), out
