// Decoding of the fixed-point outputs on the device: value = (double)(int64)
// bits / 2^e (timemachine/cpp/src/fixed_point.hpp:3-17), the per-atom energy
// and du_dl buffers summed first (wrapping, as the host sums them). Both steps
// give the same bits on either side: the integer sum is exact modulo 2^64, the
// conversion rounds to nearest, the division is by a power of two.
#pragma once

#include "nb_pair_math.cuh"

namespace tmb {

struct DecodeArgs {
    int K; // evaluations
    const unsigned long long *du_dx, *du_dp; // [n_dx], [n_dp] in all (nullptr: not requested)
    size_t n_dx, n_dp;
    int dp_columns; // 1: du_dp in (charge, sigma, epsilon) columns with exponents 36, 37, 38; 0: all 36
    const unsigned long long *du_dl, *u; // [K][N]
    int N;
    const int *error; // device error word, nullptr: none
    double *out;      // status, [K] du_dl, [K] u, du_dx, du_dp (all of them have their place)
};

__host__ __device__ __forceinline__ size_t decode_offset_dx(int K) { return 1 + 2 * (size_t)K; }

constexpr int DECODE_THREADS = 256;

// The first 2K blocks sum one evaluation's du_dl or u each, the others decode
// du_dx and du_dp element by element.
static __global__ void __launch_bounds__(DECODE_THREADS) k_decode(DecodeArgs a) {
    const double unit = 1.0 / (double)FX_EXPONENT;
    if (blockIdx.x < 2u * a.K) {
        const int k = blockIdx.x % a.K;
        const unsigned long long *row = blockIdx.x < (unsigned)a.K ? a.du_dl : a.u;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.out[0] = a.error ? (double)*a.error : 0.0;
        }
        if (row == nullptr) {
            return;
        }
        row += (size_t)k * a.N;
        unsigned long long sum = 0;
#pragma unroll 4
        for (int i = threadIdx.x; i < a.N; i += DECODE_THREADS) {
            sum += row[i];
        }
        __shared__ unsigned long long part[DECODE_THREADS / 32];
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        if ((threadIdx.x & 31) == 0) {
            part[threadIdx.x >> 5] = sum;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < DECODE_THREADS / 32; w++) {
                sum += part[w];
            }
            a.out[1 + blockIdx.x] = (double)(long long)sum * unit;
        }
        return;
    }
    double *dx = a.out + decode_offset_dx(a.K);
    double *dp = dx + a.n_dx;
    const size_t n = a.n_dx + a.n_dp;
    const size_t stride = (size_t)(gridDim.x - 2 * a.K) * DECODE_THREADS;
    for (size_t i = (size_t)(blockIdx.x - 2 * a.K) * DECODE_THREADS + threadIdx.x; i < n; i += stride) {
        if (i < a.n_dx) {
            dx[i] = (double)(long long)a.du_dx[i] * unit;
        } else {
            const size_t m = i - a.n_dx;
            const int c = a.dp_columns ? (int)(m % 3) : 0;
            dp[m] = (double)(long long)a.du_dp[m] * (c == 0 ? unit : c == 1 ? unit / 2 : unit / 4);
        }
    }
}

inline unsigned decode_grid(const DecodeArgs &a, int sms) {
    const size_t n = (a.n_dx + a.n_dp + DECODE_THREADS - 1) / DECODE_THREADS;
    const size_t most = 8 * (size_t)sms;
    return 2u * a.K + (unsigned)(n < most ? n : most);
}

} // namespace tmb
