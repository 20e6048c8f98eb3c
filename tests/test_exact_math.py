"""The EXACT mode's branch-free device arithmetic (csrc/exact_math.cuh) equals
IEEE division and square root and the portable functions bit for bit.  The
probe below is compiled like the EXACT kernels (-fmad=false) and compares on
the device over every operand, or every significand, that can occur."""
import ctypes as C
import subprocess

import pytest

PROBE = r'''
#include <cuda_runtime.h>
#include "exact_math.cuh"
typedef unsigned long long u64;

static __device__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

/* inverse of odd b modulo 2^32 (Newton on the 2-adic numbers) */
static __device__ uint32_t inverse(uint32_t b) {
    uint32_t x = b;
    for (int i = 0; i < 5; ++i) x *= 2u - b * x;
    return x;
}

static __device__ uint32_t check(int op, u64 i) {
    if (op == 0) {            /* reciprocal: every significand, three exponents */
        uint32_t m = (uint32_t)(i & 0x7fffffu), bad = 0;
        for (int e = -60; e <= 59; e += 17) {
            float b = __uint_as_float(((uint32_t)(127 + e) << 23) | m);
            bad += !same(em_recip(b), 1.0f / b) + !same(em_recip(-b), -1.0f / b);
        }
        return bad;
    }
    if (op == 1) {            /* square root and 1/sqrt: every significand, both parities */
        uint32_t m = (uint32_t)(i & 0x7fffffu), bad = 0;
        for (int e = -60; e <= 59; e += 17) {
            float x = __uint_as_float(((uint32_t)(127 + e) << 23) | m);
            bad += !same(em_sqrt(x), sqrtf(x)) + !same(em_recip(em_sqrt_normal(x)), 1.0f / sqrtf(x));
        }
        return bad;
    }
    if (op == 2) {            /* quotients next to the midpoint of two floats, for every divisor:
                                 A 2^s - N B = r with N odd and r small, s = 24 (A >= B) or 25 */
        const uint32_t B = 0x800000u + (uint32_t)i;
        const int j = __ffs((int)B) - 1;
        const uint32_t odd = B >> j, inv = inverse(odd);
        uint32_t bad = 0;
        if (j > 4) return 0;
        for (int rr = -15; rr <= 15; rr += 2)
            for (int s = 24; s <= 25; ++s) {
                const uint32_t mod = (1u << (s - j)) - 1u;
                uint32_t base = ((uint32_t)(-rr) * inv) & mod;
                for (uint32_t t = 0; t < (1u << j); ++t) {
                    u64 N = (u64)base + ((u64)t << (s - j));
                    if (s == 24) N += 1ull << 24;
                    if (!(N & 1ull) || N <= (1ull << 24) || N >= (1ull << 25)) continue;
                    u64 num = N * B + (u64)(long long)(rr * (1 << j));
                    if (num & ((1ull << s) - 1ull)) continue;
                    u64 A = num >> s;
                    if (A < 0x800000ull || A >= 0x1000000ull) continue;
                    if ((s == 24) != (A >= B)) continue;
                    float a = (float)A, b = (float)B;
                    bad += !same(em_div(a, b), a / b);
                    bad += !same(em_div(-a * 1.52587890625e-05f, b), (-a * 1.52587890625e-05f) / b);
                }
            }
        return bad;
    }
    if (op == 3) {            /* quotients of arbitrary bit patterns, special operands among them */
        u64 z = i * 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        float a = __uint_as_float((uint32_t)z), b = __uint_as_float((uint32_t)(z >> 32));
        if ((i & 15u) == 0) a = (i & 16u) ? 0.0f : -0.0f;
        if ((i & 63u) == 1) b = (i & 64u) ? 0.0f : __int_as_float(0x7f800000);
        uint32_t bad = !same(em_div(a, b), a / b) + !same(em_sqrt(a), sqrtf(a));
        /* +0 and in-range numerators over a shared reciprocal */
        float d = 0.5f + fabsf(__uint2float_rn((uint32_t)z) * 2.3283064365386963e-10f);
        bad += !same(em_quot(0.0f, d, em_recip(d)), 0.0f) + !same(em_quot(0.0f, -d, em_recip(-d)), -0.0f);
        return bad;
    }
    if (op == 4) return !same(em_log(__uint_as_float((uint32_t)i)), pm_logf(__uint_as_float((uint32_t)i)));
    if (op == 5) {            /* every uniform number of the generator */
        float u = __uint2float_rn((uint32_t)i) * 2.3283064365386963e-10f;
        float s, c, ps, pc, fi = 6.28318548f * u;
        em_sincos_azimuth(fi, &s, &c);
        pm_sincosf(fi, &ps, &pc);
        return !same(em_log_uniform(u), pm_logf(u)) + !same(s, ps) + !same(c, pc);
    }
    if (op == 6) return !same(em_exp(__uint_as_float((uint32_t)i)), pm_expf(__uint_as_float((uint32_t)i)));
    if (op == 8) {            /* every float within 2^-12 of 1 */
        float x = __uint_as_float(0x3f7ff000u + (uint32_t)i);
        return fabsf(x - 1.0f) <= 0.000244140625f && !same(em_rcp_length_near1(x), 1.0f / sqrtf(x));
    }
    float x = __uint_as_float((uint32_t)(i >> 4) * 2654435761u);
    const float ys[16] = {-1.0f, -0.5f, -2.0f, 0.0f, 1.0f, 0.333333343f, -0.833333313f, -1.0e3f,
                          2.0f, -10.0f, 0.0769230798f, -4.0f, 1e-30f, -1e30f, -3.4e38f, 1.5f};
    return !same(em_powr(x, ys[i & 15]), pm_powrf(x, ys[i & 15]));
}

static __global__ void run(int op, u64 n, u64 *bad) {
    u64 count = 0;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
        count += check(op, i);
    if (count) atomicAdd(bad, count);
}

extern "C" int probe(int op, u64 n, u64 *host_bad) {
    u64 *d = nullptr;
    if (cudaMalloc(&d, 8) != cudaSuccess) return 1;
    cudaMemset(d, 0, 8);
    run<<<152 * 8, 256>>>(op, n, d);
    int e = (int)cudaMemcpy(host_bad, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e;
}
'''


@pytest.fixture(scope='module')
def probe(cuda, tmp_path_factory):
    from pyxopto_gb300 import build
    d = tmp_path_factory.mktemp('exact_math')
    src, so = d / 'probe.cu', d / 'probe.so'
    src.write_text(PROBE)
    subprocess.run([build.nvcc_path()] + build.ARCH + ['-O3', '-std=c++17', '-fmad=false', '-I', build.CSRC,
                   '-Xcompiler', '-fPIC', '-shared', '-o', str(so), str(src)], check=True)
    lib = C.CDLL(str(so))

    def run(op, n):
        bad = C.c_ulonglong(0)
        assert lib.probe(C.c_int(op), C.c_ulonglong(n), C.byref(bad)) == 0
        return bad.value
    return run


@pytest.mark.gpu
@pytest.mark.parametrize('op,count', [
    pytest.param(0, 1 << 23, id='reciprocal'), pytest.param(1, 1 << 23, id='sqrt'),
    pytest.param(2, 1 << 23, id='quotients at midpoints'), pytest.param(3, 1 << 32, id='quotients'),
    pytest.param(4, 1 << 32, id='log'), pytest.param(5, 1 << 32, id='uniform log and azimuth'),
    pytest.param(6, 1 << 32, id='exp'), pytest.param(7, 1 << 32, id='powr'),
    pytest.param(8, 1 << 13, id='length near 1')])
def test_device_arithmetic_equals_ieee_and_portable(probe, op, count):
    assert probe(op, count) == 0
