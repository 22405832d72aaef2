// Exact direct summation (pytreegrav bruteforce.py).
//
// FP64: every operation rounded once in pytreegrav's expression order and summed over sources in
// ascending order -- the same arithmetic as the per-target CPU kernels (bruteforce.py:7-50, 86-116,
// 164-256, 259-282, 319-386), so results agree bit for bit. This is the FP64 judge the FP32 walk is scored
// against. Two forms: the pairs' terms formed by several warps and added in order by one (k_bf64_chain),
// and one target per thread (k_bf64) where such blocks fill the GPU.
//
// FP32: the fast path (the numba-cuda CudaPotentialBruteforce/CudaAccelBruteforce of cuda.py:627-796
// rebuilt): tiles of 256 sources in shared memory, two targets per thread so every broadcast source
// load feeds two interactions, rsqrt, and tile sums added into Kahan-compensated accumulators. For
// the potential and acceleration, four lanes share each pair of targets (k_bf32_split), the two
// targets are computed with paired f32x2 arithmetic, and the sources are narrowed once (k_bf32_prep).
#include <cuda_pipeline.h>

#include <algorithm>

#include "tg_common.cuh"

namespace tg {

enum { BF_POT = 1, BF_ACC = 2, BF_TID = 4 };

// kernel.py:5-75 in FP64 with single rounding per operation.
__device__ __forceinline__ double force_kernel_x(double r, double h) {
    if (r > h) return ddiv(1.0, dmul(dmul(r, r), r));
    double hinv = ddiv(1.0, h);
    double q = dmul(r, hinv);
    if (q <= 0.5)
        return dmul(dmul(dmul(dadd(10.666666666666666666, dmul(dmul(q, q), dadd(-38.4, dmul(32.0, q)))), hinv), hinv),
                    hinv);
    double t = dsub(dadd(dsub(21.333333333333, dmul(48.0, q)), dmul(dmul(38.4, q), q)),
                    dmul(dmul(dmul(10.666666666667, q), q), q));
    t = dsub(t, ddiv(0.066666666667, dmul(dmul(q, q), q)));
    return dmul(dmul(dmul(t, hinv), hinv), hinv);
}

__device__ __forceinline__ double tidal_kernel_x(double r, double h) {
    if (r > h) {
        double r2 = dmul(r, r);
        return ddiv(3.0, dmul(dmul(r2, r2), r));
    }
    double hinv = ddiv(1.0, h);
    double hinv2 = dmul(hinv, hinv);
    double hinv5 = dmul(dmul(hinv2, hinv2), hinv);
    double q = dmul(r, hinv);
    if (q <= 0.5) return dmul(dsub(76.8, dmul(96.0, q)), hinv5);
    double qinv = ddiv(1.0, q);
    double qinv3 = dmul(dmul(qinv, qinv), qinv);
    double t = dadd(dsub(dmul(48.0, qinv), 76.8), dmul(32.0, q));
    t = dsub(t, dmul(dmul(dmul(0.2, qinv3), qinv), qinv));
    return dmul(t, hinv5);
}

__device__ __forceinline__ double potential_kernel_x(double r, double h) {
    if (h == 0.0) return ddiv(-1.0, r);
    double hinv = ddiv(1.0, h);
    double q = dmul(r, hinv);
    if (q <= 0.5) {
        double in = dsub(dmul(6.4, q), 9.6);
        in = dadd(5.33333333333333333, dmul(dmul(q, q), in));
        return dmul(dadd(-2.8, dmul(dmul(q, q), in)), hinv);
    }
    if (q <= 1) {
        double in = dsub(9.6, dmul(2.1333333333333333333333, q));
        in = dadd(-16.0, dmul(q, in));
        in = dadd(10.666666666666666666666, dmul(q, in));
        double t = dadd(dadd(-3.2, ddiv(0.066666666666666666666, q)), dmul(dmul(q, q), in));
        return dmul(t, hinv);
    }
    return ddiv(-1.0, r);
}

constexpr int BF64_THREADS = 128;

template <int FIELDS, bool MUTUAL>
__global__ void __launch_bounds__(BF64_THREADS) k_bf64(const double *pt, const double *ht, int64_t nt,
                                                       const double *ps, const double *ms, const double *hs,
                                                       int64_t ns, double G, double *out, int W) {
    __shared__ double sx[BF64_THREADS], sy[BF64_THREADS], sz[BF64_THREADS], sm[BF64_THREADS], sh[BF64_THREADS];
    int64_t i = (int64_t)blockIdx.x * BF64_THREADS + threadIdx.x;
    bool valid = i < nt;
    double x = valid ? pt[3 * i] : 0.0, y = valid ? pt[3 * i + 1] : 0.0, z = valid ? pt[3 * i + 2] : 0.0;
    double hti = valid ? ht[i] : 0.0;
    double phi = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0;
    double T0 = 0, T1 = 0, T2 = 0, T4 = 0, T5 = 0, T8 = 0;
    for (int64_t base = 0; base < ns; base += BF64_THREADS) {
        int64_t j = base + threadIdx.x;
        if (j < ns) {
            sx[threadIdx.x] = ps[3 * j];
            sy[threadIdx.x] = ps[3 * j + 1];
            sz[threadIdx.x] = ps[3 * j + 2];
            sm[threadIdx.x] = ms[j];
            sh[threadIdx.x] = hs[j];
        }
        __syncthreads();
        int lim = (int)((ns - base) < BF64_THREADS ? (ns - base) : BF64_THREADS);
        if (valid) {
            for (int k = 0; k < lim; k++) {
                int64_t jj = base + k;
                if (MUTUAL && jj == i) continue;
                double m = sm[k];
                if (FIELDS & BF_POT) {
                    double d0 = dsub(x, sx[k]), d1 = dsub(y, sy[k]), d2 = dsub(z, sz[k]);
                    double r = __dsqrt_rn(dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2)));
                    if (MUTUAL) {
                        double h = pymax(hti, sh[k]);
                        if (r < h) phi = dadd(phi, dmul(m, potential_kernel_x(r, h)));
                        else if (r > 0) phi = dsub(phi, ddiv(m, r));
                    } else if (r != 0) {
                        double h = pymax(sh[k], hti);
                        if (r < h) phi = dadd(phi, dmul(m, potential_kernel_x(r, h)));
                        else phi = dsub(phi, ddiv(m, r));
                    }
                }
                if (FIELDS & (BF_ACC | BF_TID)) {
                    double d0 = dsub(sx[k], x), d1 = dsub(sy[k], y), d2 = dsub(sz[k], z);
                    double r2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
                    if (r2 == 0) continue;
                    double r = __dsqrt_rn(r2);
                    double h = pymax(hti, sh[k]);
                    if (FIELDS & BF_ACC) {
                        if (r < h) {
                            double km = dmul(force_kernel_x(r, h), m);
                            a0 = dadd(a0, dmul(km, d0));
                            a1 = dadd(a1, dmul(km, d1));
                            a2 = dadd(a2, dmul(km, d2));
                        } else {
                            double mf = dmul(m, ddiv(1.0, dmul(r2, r)));
                            a0 = dadd(a0, dmul(mf, d0));
                            a1 = dadd(a1, dmul(mf, d1));
                            a2 = dadd(a2, dmul(mf, d2));
                        }
                    }
                    if (FIELDS & BF_TID) {
                        double K, Q;
                        if (r < h) {
                            K = dmul(m, force_kernel_x(r, h));
                            Q = dmul(m, tidal_kernel_x(r, h));
                        } else {
                            K = ddiv(m, dmul(r, r2));
                            Q = ddiv(dmul(3.0, K), r2);
                        }
                        T0 = dadd(T0, dsub(dmul(dmul(Q, d0), d0), K));
                        T4 = dadd(T4, dsub(dmul(dmul(Q, d1), d1), K));
                        T8 = dadd(T8, dsub(dmul(dmul(Q, d2), d2), K));
                        T1 = dadd(T1, dmul(dmul(Q, d0), d1));
                        T2 = dadd(T2, dmul(dmul(Q, d0), d2));
                        T5 = dadd(T5, dmul(dmul(Q, d1), d2));
                    }
                }
            }
        }
        __syncthreads();
    }
    if (!valid) return;
    double *o = out + i * W;
    int k = 0;
    if (FIELDS & BF_POT) o[k++] = dmul(G, phi);
    if (FIELDS & BF_ACC) {
        o[k] = dmul(G, a0);
        o[k + 1] = dmul(G, a1);
        o[k + 2] = dmul(G, a2);
        k += 3;
    }
    if (FIELDS & BF_TID) {
        double v[9] = {T0, T1, T2, T1, T4, T5, T2, T5, T8};
        for (int q = 0; q < 9; q++) o[k + q] = dmul(G, v[q]);
    }
}

// Few targets: k_bf64 gives a target one thread, and its FP64 stream (~33 instructions per source, one
// issued every ~76 cycles whatever the number of active lanes) is then the kernel's length: 700
// targets are 22 warps on 608 sub-partitions. Here a block takes T targets and cuts the stream in
// two: seven warps form the pairs' terms, lane = source, 32 sources of one target at a time, into a
// ring of tiles in shared memory, and the eighth adds the terms, lane = (target, component), one
// FP64 add per source. Every sum takes the same terms in the same ascending order as k_bf64's, so the
// results are the same bits: a pair that k_bf64 skips adds -0.0, the exact identity of a sum.
// The adder needs one instruction per source and block, the others ~30 T / 32: T is the targets'
// number over the SMs, at most what fills the adder's lanes. Two items per producer and stage keep the
// pipeline's fill short against 700 sources. The softening tests run on the integer units, and 1 / x is
// __drcp_rn, the same correctly rounded value as the division.
// Acceleration: 700 bodies' own 860 -> 53 us (FP64 pipe 64 % busy; floor ~28 us of pairs); 2000 sources
// and 100 targets 2499 -> 116 us, 2000 targets 2498 -> 318, 1e4 2499 -> 1402, 2e4 4608 -> 2760.
constexpr int BFC_PRODUCERS = 7, BFC_THREADS = 32 * (BFC_PRODUCERS + 1);
constexpr int BFC_UNITS = 2;                                 // (tile, target) items per producer and stage
constexpr int BFC_STAGE = BFC_PRODUCERS * BFC_UNITS;         // items per stage
constexpr int BFC_ROW = 33;                                  // doubles per chain and tile (odd: no bank conflicts)
template <int FIELDS>
__host__ __device__ constexpr int bfc_comps() {
    return ((FIELDS & BF_POT) ? 1 : 0) + ((FIELDS & BF_ACC) ? 3 : 0) + ((FIELDS & BF_TID) ? 6 : 0);
}
// k_bf64 is the faster form only where its blocks of 128 targets, one per SM, fill their last wave. Its
// time goes by whole waves (2000 sources, acceleration: 2.31 ms each), this form's by targets and with
// the adder (60000 targets 7.80 ms, 1.10 times as much per target as a full wave; potential 1.11,
// tidal tensor 1.06). With every field (ten components, three targets per block) this form is the
// faster one throughout: 18.0 ms for 60000 targets against 20.5 for three full waves (58368).
constexpr int64_t BFC_MAX_SOURCES = 1 << 29;  // (tile, target) items are counted in 32 bits
template <int FIELDS>
static bool bf64_chain_better(int64_t nt, int64_t ns) {
    if (ns > BFC_MAX_SOURCES) return false;
    if (FIELDS == (BF_POT | BF_ACC | BF_TID)) return true;
    const int64_t wave = (int64_t)num_sms() * BF64_THREADS, waves = (nt + wave - 1) / wave;
    return 100 * nt < 92 * waves * wave;
}
// Tiles of the ring: a stage writes at most BFC_STAGE / T + 2 tiles while as many are summed.
__host__ __device__ inline int bfc_ring(int T) { return 2 * BFC_STAGE / T + 3; }

// Order key of a softening length: a signed integer of the same order as the value (-0.0 as +0.0), the
// least for NaN, which no distance is below.
__device__ __forceinline__ long long soft_key(double h) {
    const long long b = __double_as_longlong(h);
    const long long mag = b & 0x7fffffffffffffffll;
    if (mag > 0x7ff0000000000000ll) return (long long)0x8000000000000000ull;
    return b < 0 ? -mag : mag;
}
// r < pymax(a, b) for a distance r (>= 0 or NaN), decided on the integer units: pymax is NaN when a
// is, and a when b is.
__device__ __forceinline__ bool below_max(double r, long long ka, long long kb) {
    const long long none = (long long)0x8000000000000000ull;
    const long long k = ka == none ? none : (kb > ka ? kb : ka);
    return (__double_as_longlong(r) & 0x7fffffffffffffffll) < k;
}

template <int FIELDS, bool MUTUAL>
__global__ void __launch_bounds__(BFC_THREADS) k_bf64_chain(const double *pt, const double *ht, int64_t nt,
                                                            const double *ps, const double *ms, const double *hs,
                                                            int64_t ns, int T, double G, double *out, int W) {
    extern __shared__ double bfc_ring_mem[];  // [ring][T * C][BFC_ROW]
    constexpr int C = bfc_comps<FIELDS>();
    __shared__ double tx[32], ty[32], tz[32], th[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ring = bfc_ring(T);
    const int64_t t0 = (int64_t)blockIdx.x * T;
    if (threadIdx.x < T) {
        const int64_t i = t0 + threadIdx.x < nt ? t0 + threadIdx.x : nt - 1;
        tx[threadIdx.x] = pt[3 * i];
        ty[threadIdx.x] = pt[3 * i + 1];
        tz[threadIdx.x] = pt[3 * i + 2];
        th[threadIdx.x] = ht[i];
    }
    __syncthreads();
    const int ntiles = (int)((ns + 31) / 32), nitems = ntiles * T;  // ns <= BFC_MAX_SOURCES
    const int nstages = (nitems + BFC_STAGE - 1) / BFC_STAGE;
    double sum = 0.0;  // the adder's chain
    int consumed = 0;  // tiles added so far
    for (int st = 0; st <= nstages; st++) {
        if (w < BFC_PRODUCERS) {
#pragma unroll 1
            for (int u = 0; u < BFC_UNITS; u++) {
                const int item = st * BFC_STAGE + w * BFC_UNITS + u;
                if (item >= nitems) break;
                const int tile = item / T, t = item - tile * T;
                const int64_t j = (int64_t)tile * 32 + lane;
                double term[C];
#pragma unroll
                for (int c = 0; c < C; c++) term[c] = -0.0;
                if (j < ns && !(MUTUAL && j == t0 + t)) {
                    const double m = ms[j], hj = hs[j], hti = th[t];
                    const double d0 = dsub(ps[3 * j], tx[t]), d1 = dsub(ps[3 * j + 1], ty[t]);
                    const double d2 = dsub(ps[3 * j + 2], tz[t]);
                    const double r2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
                    const double r = __dsqrt_rn(r2);
                    const long long kt = soft_key(hti), kj = soft_key(hj);
                    if (FIELDS & BF_POT) {  // phi - m / r is phi + (-(m / r))
                        const bool in = MUTUAL ? below_max(r, kt, kj) : below_max(r, kj, kt);
                        // mutual: r > 0 outside the softening; else r != 0 (true of NaN too)
                        const long long rb = __double_as_longlong(r) & 0x7fffffffffffffffll;
                        if (MUTUAL) {
                            if (in) term[0] = dmul(m, potential_kernel_x(r, pymax(hti, hj)));
                            else if (rb > 0 && rb <= 0x7ff0000000000000ll) term[0] = -ddiv(m, r);
                        } else if (rb != 0) {
                            if (in) term[0] = dmul(m, potential_kernel_x(r, pymax(hj, hti)));
                            else term[0] = -ddiv(m, r);
                        }
                    }
                    if ((FIELDS & (BF_ACC | BF_TID)) && (__double_as_longlong(r2) << 1) != 0) {
                        const bool in = below_max(r, kt, kj);
                        const double h = in ? pymax(hti, hj) : 0.0;
                        double *p = term + ((FIELDS & BF_POT) ? 1 : 0);
                        if (FIELDS & BF_ACC) {
                            // 1 / x correctly rounded is the same value from __drcp_rn
                            const double mf = in ? dmul(force_kernel_x(r, h), m) : dmul(m, __drcp_rn(dmul(r2, r)));
                            p[0] = dmul(mf, d0);
                            p[1] = dmul(mf, d1);
                            p[2] = dmul(mf, d2);
                            p += 3;
                        }
                        if (FIELDS & BF_TID) {
                            double K, Q;
                            if (in) {
                                K = dmul(m, force_kernel_x(r, h));
                                Q = dmul(m, tidal_kernel_x(r, h));
                            } else {
                                K = ddiv(m, dmul(r, r2));
                                Q = ddiv(dmul(3.0, K), r2);
                            }
                            const double q0 = dmul(Q, d0), q1 = dmul(Q, d1);
                            p[0] = dsub(dmul(q0, d0), K);
                            p[1] = dmul(q0, d1);
                            p[2] = dmul(q0, d2);
                            p[3] = dsub(dmul(q1, d1), K);
                            p[4] = dmul(q1, d2);
                            p[5] = dsub(dmul(dmul(Q, d2), d2), K);
                        }
                    }
                }
                double *slot = bfc_ring_mem + ((tile % ring) * T + t) * (C * BFC_ROW) + lane;
#pragma unroll
                for (int c = 0; c < C; c++) slot[c * BFC_ROW] = term[c];
            }
        } else {
            // the tiles that the earlier stages completed
            const int ready = min(st * BFC_STAGE / T, ntiles);
            if (lane < T * C)
                for (; consumed < ready; consumed++) {
                    const double *row = bfc_ring_mem + (consumed % ring) * (T * C * BFC_ROW) + lane * BFC_ROW;
#pragma unroll 16
                    for (int k = 0; k < 32; k++) sum = dadd(sum, row[k]);
                }
        }
        __syncthreads();
    }
    if (w == BFC_PRODUCERS && lane < T * C) {
        const int t = lane / C;
        int c = lane - t * C;
        if (t0 + t >= nt) return;
        double *o = out + (t0 + t) * W;
        const double v = dmul(G, sum);
        if (FIELDS & BF_POT) {
            if (c == 0) {
                o[0] = v;
                return;
            }
            c--;
            o++;
        }
        if (FIELDS & BF_ACC) {
            if (c < 3) {
                o[c] = v;
                return;
            }
            c -= 3;
            o += 3;
        }
        // xx xy xz yy yz zz into the symmetric 3x3
        const int row = c < 3 ? 0 : (c < 5 ? 1 : 2), col = c < 3 ? c : (c < 5 ? c - 2 : 2);
        o[3 * row + col] = v;
        o[3 * col + row] = v;
    }
}

// ---------------------------------------------------------------------------------------------
constexpr int BF32_THREADS = 256;
constexpr int BF32_TPT = 2;

template <int FIELDS>
__device__ __forceinline__ void bf32_pair(float m, float hs, float ht, float dx, float dy, float dz, bool skip,
                                          float *p) {
    float r2 = dx * dx + dy * dy + dz * dz;
    if (skip || !(r2 > 0.f)) return;
    float rinv = rsqrtf(r2);
    float r = r2 * rinv;
    float h = hs > ht ? hs : ht;
    float K, Q = 0.f;
    if (r < h) {
        float hinv = 1.f / h, q = r * hinv, h3 = hinv * hinv * hinv;
        if (FIELDS & BF_POT) {
            float pk;
            if (q <= 0.5f) pk = (-2.8f + q * q * (5.333333333f + q * q * (6.4f * q - 9.6f))) * hinv;
            else pk = (-3.2f + 0.0666666667f / q + q * q * (10.66666667f + q * (-16.0f + q * (9.6f - 2.133333333f * q)))) * hinv;
            p[0] += m * pk;
        }
        if (q <= 0.5f) K = (10.66666667f + q * q * (-38.4f + 32.0f * q)) * h3;
        else K = (21.333333333f - 48.0f * q + 38.4f * q * q - 10.666666667f * q * q * q - 0.066666666667f / (q * q * q)) * h3;
        K *= m;
        if (FIELDS & BF_TID) {
            float h5 = h3 * hinv * hinv;
            float tk;
            if (q <= 0.5f) tk = (76.8f - 96.0f * q) * h5;
            else {
                float qi = 1.f / q, qi3 = qi * qi * qi;
                tk = (48.0f * qi - 76.8f + 32.0f * q - 0.2f * qi3 * qi * qi) * h5;
            }
            Q = m * tk;
        }
    } else {
        float rinv2 = rinv * rinv, mr = m * rinv;
        if (FIELDS & BF_POT) p[0] -= mr;
        K = mr * rinv2;
        if (FIELDS & BF_TID) Q = 3.f * K * rinv2;
    }
    if (FIELDS & BF_ACC) {
        p[1] += K * dx;
        p[2] += K * dy;
        p[3] += K * dz;
    }
    if (FIELDS & BF_TID) {
        float qx = Q * dx, qy = Q * dy;
        p[4] += qx * dx - K;
        p[5] += qx * dy;
        p[6] += qx * dz;
        p[7] += qy * dy - K;
        p[8] += qy * dz;
        p[9] += Q * dz * dz - K;
    }
}

template <int FIELDS, bool MUTUAL>
__global__ void __launch_bounds__(BF32_THREADS) k_bf32(const double *pt, const double *ht, int64_t nt,
                                                       const double *ps, const double *ms, const double *hs,
                                                       int64_t ns, double G, double *out, int W) {
    __shared__ float4 spos[BF32_THREADS];
    __shared__ float sh[BF32_THREADS];
    float tx[BF32_TPT], ty[BF32_TPT], tz[BF32_TPT], th[BF32_TPT];
    int64_t ti[BF32_TPT];
    float S[BF32_TPT][10], C[BF32_TPT][10];
#pragma unroll
    for (int u = 0; u < BF32_TPT; u++) {
        ti[u] = ((int64_t)blockIdx.x * BF32_TPT + u) * BF32_THREADS + threadIdx.x;
        int64_t i = ti[u] < nt ? ti[u] : 0;
        tx[u] = (float)pt[3 * i];
        ty[u] = (float)pt[3 * i + 1];
        tz[u] = (float)pt[3 * i + 2];
        th[u] = (float)ht[i];
#pragma unroll
        for (int c = 0; c < 10; c++) S[u][c] = C[u][c] = 0.f;
    }
    for (int64_t base = 0; base < ns; base += BF32_THREADS) {
        int64_t j = base + threadIdx.x;
        if (j < ns) {
            spos[threadIdx.x] = make_float4((float)ps[3 * j], (float)ps[3 * j + 1], (float)ps[3 * j + 2], (float)ms[j]);
            sh[threadIdx.x] = (float)hs[j];
        }
        __syncthreads();
        int lim = (int)((ns - base) < BF32_THREADS ? (ns - base) : BF32_THREADS);
        float P[BF32_TPT][10];
#pragma unroll
        for (int u = 0; u < BF32_TPT; u++)
#pragma unroll
            for (int c = 0; c < 10; c++) P[u][c] = 0.f;
        for (int k = 0; k < lim; k++) {
            float4 s = spos[k];
            float hsk = sh[k];
#pragma unroll
            for (int u = 0; u < BF32_TPT; u++) {
                bool skip = MUTUAL && (base + k == ti[u]);
                bf32_pair<FIELDS>(s.w, hsk, th[u], s.x - tx[u], s.y - ty[u], s.z - tz[u], skip, P[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < BF32_TPT; u++)
#pragma unroll
            for (int c = 0; c < 10; c++) {
                float yv = P[u][c] - C[u][c];
                float tv = S[u][c] + yv;
                C[u][c] = (tv - S[u][c]) - yv;
                S[u][c] = tv;
            }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < BF32_TPT; u++) {
        if (ti[u] >= nt) continue;
        double *o = out + ti[u] * W;
        double v[10];
        for (int c = 0; c < 10; c++) v[c] = G * ((double)S[u][c] - (double)C[u][c]);
        int k = 0;
        if (FIELDS & BF_POT) o[k++] = v[0];
        if (FIELDS & BF_ACC) {
            o[k] = v[1];
            o[k + 1] = v[2];
            o[k + 2] = v[3];
            k += 3;
        }
        if (FIELDS & BF_TID) {
            double tv[9] = {v[4], v[5], v[6], v[5], v[7], v[8], v[6], v[8], v[9]};
            for (int q = 0; q < 9; q++) o[k + q] = tv[q];
        }
    }
}

// Potential and/or acceleration, the main FP32 form: BF32S_LANES lanes share each pair of targets,
// lane q of the group taking the sources k = q (mod BF32S_LANES) of every tile, so a target set of 1e5
// still fills the GPU; the lanes' Kahan-compensated sums (compensated once per tile) are combined at
// the end by a fixed pattern of shuffles (deterministic). The two targets are computed together
// with paired f32x2 arithmetic for every source outside both softening lengths (with a 1e-5 margin)
// and not coincident; any other source takes bf32_pair for each target.
//
// Bound by issue slots and the FP32 pipe (12 operations and an rsqrt per pair of particles; 0.75 ms at
// 5e4 x 5e4), and by the chain of one source's operations where the targets are few. For that:
//   * BF32S_UNROLL sources at a time, their distances first: the chains overlap (5e4 sources, acceleration:
//     1000 targets 778 us at 2, 504 at 4, 433 at 8 and 411 at 16, where 1e5 targets lose 30 % to spills);
//   * one test per distance against a bound beyond which no source of the tile (its largest h^2 comes
//     from k_bf32_prep) and neither target is softened, instead of the exact test, which only a batch
//     that fails the bound takes, source by source;
//   * the sources are narrowed to FP32 once (k_bf32_prep), not by every block for every tile, which kept the
//     FP64 pipe busy with conversions.
// 5e4 sources, acceleration, before and after: 1000 targets 1330 -> 433 us, 2e4 1645 -> 761, 50001
// 2262 -> 1403, 1e5 4271 -> 2461. Measured and dropped: two pairs of targets per lane (50001: 1458;
// 1e5: 2686; 1000: 761), each staged value duplicated for the paired operands (1e5: 2795; shared-memory
// reads return 4 words per lane and cycle), scalar subtractions and products (1e5: 2644).
constexpr int BF32S_THREADS = 128;
constexpr int BF32S_BLOCKS_PER_SM = 4;  // at most 128 registers
constexpr int BF32S_LANES = 4;
constexpr int BF32S_TILE = 256;  // sources per tile
constexpr int BF32S_UNROLL = 8;
constexpr int BF32S_PAIRS = BF32S_THREADS / BF32S_LANES;  // pairs of targets per block

typedef unsigned long long bf2;
__device__ __forceinline__ bf2 bf2_pack(float a, float b) {
    bf2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void bf2_unpack(bf2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ bf2 bf2_fma(bf2 a, bf2 b, bf2 c) {
    bf2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ bf2 bf2_mul(bf2 a, bf2 b) {
    bf2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ bf2 bf2_sub(bf2 a, bf2 b) {
    bf2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ float bf32_rsqrt_normal(float x) {  // rsqrtf's value for a normal x > 0
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Sources in FP32, (x, y, z, m) and (h, h^2), and each tile's largest h^2 (infinite when one is NaN, so that
// the tile's sources all take the exact test).
__global__ void __launch_bounds__(BF32S_TILE) k_bf32_prep(const double *ps, const double *ms, const double *hs,
                                                          int64_t ns, float4 *src, float2 *soft, float *tile_h2) {
    __shared__ float wmax[BF32S_TILE / 32];
    const int64_t j = (int64_t)blockIdx.x * BF32S_TILE + threadIdx.x;
    float h2 = 0.f;
    if (j < ns) {
        const float h = d2f(hs[j]);
        h2 = h * h;
        src[j] = make_float4(d2f(ps[3 * j]), d2f(ps[3 * j + 1]), d2f(ps[3 * j + 2]), d2f(ms[j]));
        soft[j] = make_float2(h, h2);
        if (!(h2 == h2)) h2 = INFINITY;
    }
    for (int o = 16; o; o >>= 1) h2 = fmaxf(h2, __shfl_xor_sync(FULL, h2, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = h2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < BF32S_TILE / 32; w++) h2 = fmaxf(h2, wmax[w]);
        tile_h2[blockIdx.x] = h2;
    }
}

template <int FIELDS, bool MUTUAL>
__global__ void __launch_bounds__(BF32S_THREADS, BF32S_BLOCKS_PER_SM) k_bf32_split(
    const double *pt, const double *ht, int64_t nt, const float4 *src, const float2 *soft, const float *tile_h2,
    int64_t ns, double G, double *out, int W) {
    __shared__ float4 spos[2][BF32S_TILE];
    __shared__ float2 ssoft[2][BF32S_TILE];
    constexpr int C0 = (FIELDS & BF_POT) ? 0 : 1, C1 = (FIELDS & BF_ACC) ? 4 : 1;  // components used
    const int q = threadIdx.x % BF32S_LANES;
    const int64_t t0 = 2 * ((int64_t)blockIdx.x * BF32S_PAIRS + threadIdx.x / BF32S_LANES);  // targets t0, t0 + 1
    float tx[2], ty[2], tz[2], th[2], th2[2], th2max = 0.f;
    float S[2][4], C[2][4];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int64_t i = t0 + u < nt ? t0 + u : 0;
        tx[u] = d2f(pt[3 * i]);
        ty[u] = d2f(pt[3 * i + 1]);
        tz[u] = d2f(pt[3 * i + 2]);
        th[u] = d2f(ht[i]);
        th2[u] = th[u] * th[u];
        th2max = fmaxf(th2max, th2[u] == th2[u] ? th2[u] : INFINITY);
#pragma unroll
        for (int c = 0; c < 4; c++) S[u][c] = C[u][c] = 0.f;
    }
    const bf2 TX = bf2_pack(tx[0], tx[1]), TY = bf2_pack(ty[0], ty[1]), TZ = bf2_pack(tz[0], tz[1]);
    const int64_t ntiles = (ns + BF32S_TILE - 1) / BF32S_TILE;
    auto stage = [&](int64_t tile, int buf) {  // the next tile is copied while one is summed
        for (int i = threadIdx.x; i < BF32S_TILE; i += BF32S_THREADS) {
            const int64_t j = tile * BF32S_TILE + i;
            if (j < ns) {
                __pipeline_memcpy_async(&spos[buf][i], src + j, sizeof(float4));
                __pipeline_memcpy_async(&ssoft[buf][i], soft + j, sizeof(float2));
            }
        }
        __pipeline_commit();
    };
    stage(0, 0);
    for (int64_t tile = 0; tile < ntiles; tile++) {
        const int buf = (int)(tile & 1);
        stage(tile + 1, buf ^ 1);  // past the last tile: nothing to copy
        __pipeline_wait_prior(1);
        __syncthreads();
        const int64_t base = tile * BF32S_TILE;
        const int lim = (int)((ns - base) < BF32S_TILE ? (ns - base) : BF32S_TILE);
        // beyond this squared distance no pair of the tile is softened, and r2 is a normal number
        const float far2 = fmaxf(fmaxf(tile_h2[tile], th2max) * 1.00001f, 1.2e-38f);
        bf2 ph = 0, ax = 0, ay = 0, az = 0;  // the two targets' tile sums (bit pattern 0 is +0.0f, +0.0f)
        float P[2][10];
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int c = 0; c < 10; c++) P[u][c] = 0.f;
        auto add_far = [&](float m, bf2 dx, bf2 dy, bf2 dz, float ri0, float ri1) {
            const bf2 rinv = bf2_pack(ri0, ri1);
            const bf2 mr = bf2_mul(bf2_pack(m, m), rinv);
            if (FIELDS & BF_POT) ph = bf2_sub(ph, mr);
            if (FIELDS & BF_ACC) {
                const bf2 K = bf2_mul(mr, bf2_mul(rinv, rinv));
                ax = bf2_fma(K, dx, ax);
                ay = bf2_fma(K, dy, ay);
                az = bf2_fma(K, dz, az);
            }
        };
        // one source with the exact test
        auto one = [&](int k) {
            const float4 s = spos[buf][k];
            const float2 hk = ssoft[buf][k];
            const bf2 dx = bf2_sub(bf2_pack(s.x, s.x), TX), dy = bf2_sub(bf2_pack(s.y, s.y), TY);
            const bf2 dz = bf2_sub(bf2_pack(s.z, s.z), TZ);
            float r20, r21;
            bf2_unpack(bf2_fma(dz, dz, bf2_fma(dy, dy, bf2_mul(dx, dx))), r20, r21);
            const float lim0 = fmaxf(hk.y, th2[0]) * 1.00001f, lim1 = fmaxf(hk.y, th2[1]) * 1.00001f;
            bool slow = !(r20 > lim0) || !(r21 > lim1) || !(r20 > 0.f) || !(r21 > 0.f);
            if (MUTUAL) slow = slow || base + k == t0 || base + k == t0 + 1;
            if (slow) {
                float d[3][2];
                bf2_unpack(dx, d[0][0], d[0][1]);
                bf2_unpack(dy, d[1][0], d[1][1]);
                bf2_unpack(dz, d[2][0], d[2][1]);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const bool skip = MUTUAL && (base + k == t0 + u);
                    bf32_pair<FIELDS>(s.w, hk.x, th[u], d[0][u], d[1][u], d[2][u], skip, P[u]);
                }
            } else {
                add_far(s.w, dx, dy, dz, rsqrtf(r20), rsqrtf(r21));
            }
        };
        int k = q;
        for (; k + (BF32S_UNROLL - 1) * BF32S_LANES < lim; k += BF32S_UNROLL * BF32S_LANES) {
            bf2 dx[BF32S_UNROLL], dy[BF32S_UNROLL], dz[BF32S_UNROLL];
            float r2[BF32S_UNROLL][2], m[BF32S_UNROLL];
            bool far = true;
#pragma unroll
            for (int e = 0; e < BF32S_UNROLL; e++) {
                const float4 s = spos[buf][k + e * BF32S_LANES];
                m[e] = s.w;
                dx[e] = bf2_sub(bf2_pack(s.x, s.x), TX);
                dy[e] = bf2_sub(bf2_pack(s.y, s.y), TY);
                dz[e] = bf2_sub(bf2_pack(s.z, s.z), TZ);
                bf2_unpack(bf2_fma(dz[e], dz[e], bf2_fma(dy[e], dy[e], bf2_mul(dx[e], dx[e]))), r2[e][0], r2[e][1]);
                far = far && r2[e][0] > far2 && r2[e][1] > far2;
            }
            if (far) {
#pragma unroll
                for (int e = 0; e < BF32S_UNROLL; e++)
                    add_far(m[e], dx[e], dy[e], dz[e], bf32_rsqrt_normal(r2[e][0]), bf32_rsqrt_normal(r2[e][1]));
            } else {
#pragma unroll 1
                for (int e = 0; e < BF32S_UNROLL; e++) one(k + e * BF32S_LANES);
            }
        }
#pragma unroll 1
        for (; k < lim; k += BF32S_LANES) one(k);
        const bf2 fast[4] = {ph, ax, ay, az};
#pragma unroll
        for (int c = C0; c < C1; c++) {
            float a0, a1;
            bf2_unpack(fast[c], a0, a1);
            P[0][c] += a0;
            P[1][c] += a1;
        }
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int c = C0; c < C1; c++) {
                const float yv = P[u][c] - C[u][c];
                const float tv = S[u][c] + yv;
                C[u][c] = (tv - S[u][c]) - yv;
                S[u][c] = tv;
            }
        __syncthreads();
    }
    __pipeline_wait_prior(0);
    // the group's lanes combined in double, the same fixed pattern on every lane
#pragma unroll
    for (int u = 0; u < 2; u++) {
        double v[4];
#pragma unroll
        for (int c = C0; c < C1; c++) {
            v[c] = (double)S[u][c] - (double)C[u][c];
#pragma unroll
            for (int o = 1; o < BF32S_LANES; o <<= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
        }
        if (q != 0 || t0 + u >= nt) continue;
        double *o = out + (t0 + u) * W;
        int k = 0;
        if (FIELDS & BF_POT) o[k++] = G * v[0];
        if (FIELDS & BF_ACC) {
            o[k] = G * v[1];
            o[k + 1] = G * v[2];
            o[k + 2] = G * v[3];
        }
    }
}

template <int FIELDS, bool MUTUAL>
static tg_status launch_bf(int precision, const double *pt, const double *ht, int64_t nt, const double *ps,
                      const double *ms, const double *hs, int64_t ns, double G, double *out, int W, cudaStream_t st) {
    if (precision == TG_FP64 && bf64_chain_better<FIELDS>(nt, ns)) {
        constexpr int C = bfc_comps<FIELDS>(), most = 32 / C;
        // as many targets per block as let every SM have the same number of blocks
        const int64_t sms = num_sms();
        const int T = div_up(nt, sms * div_up(nt, sms * most));
        const size_t smem = sizeof(double) * (size_t)bfc_ring(T) * T * C * BFC_ROW;
        auto kern = k_bf64_chain<FIELDS, MUTUAL>;
        TG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        { kern<<<div_up(nt, T), BFC_THREADS, smem, st>>>(pt, ht, nt, ps, ms, hs, ns, T, G, out, W); tg::note_launch(); }
    } else if (precision == TG_FP64) {
        { k_bf64<FIELDS, MUTUAL><<<div_up(nt, BF64_THREADS), BF64_THREADS, 0, st>>>(pt, ht, nt, ps, ms, hs, ns, G, out, W); tg::note_launch(); }
    } else if constexpr ((FIELDS & BF_TID) == 0) {
        const int64_t ntiles = div_up(ns, BF32S_TILE);
        DevArray<float4> src(st);
        DevArray<float2> soft(st);
        DevArray<float> tile_h2(st);
        TG_CUDA(src.alloc(ns));
        TG_CUDA(soft.alloc(ns));
        TG_CUDA(tile_h2.alloc(ntiles));
        if (ntiles > 0) { k_bf32_prep<<<(unsigned)ntiles, BF32S_TILE, 0, st>>>(ps, ms, hs, ns, src.p, soft.p, tile_h2.p); tg::note_launch(); }
        { k_bf32_split<FIELDS, MUTUAL><<<div_up(nt, 2 * BF32S_PAIRS), BF32S_THREADS, 0, st>>>(pt, ht, nt, src.p, soft.p,
                                                                                         tile_h2.p, ns, G, out, W); tg::note_launch(); }
    } else {
        { k_bf32<FIELDS, MUTUAL><<<div_up(nt, BF32_THREADS * BF32_TPT), BF32_THREADS, 0, st>>>(pt, ht, nt, ps, ms, hs, ns,
                                                                                           G, out, W); tg::note_launch(); }
    }
    return TG_OK;
}

template <bool MUTUAL>
static tg_status dispatch_bf(int fields, int precision, const double *pt, const double *ht, int64_t nt, const double *ps,
                        const double *ms, const double *hs, int64_t ns, double G, double *out, int W, cudaStream_t st) {
    switch (fields) {
        case 1: return launch_bf<1, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        case 2: return launch_bf<2, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        case 3: return launch_bf<3, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        case 4: return launch_bf<4, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        case 5: return launch_bf<5, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        case 6: return launch_bf<6, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
        default: return launch_bf<7, MUTUAL>(precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st);
    }
}

tg_status run_bruteforce(const double *pt, const double *ht, int64_t nt, const double *ps, const double *ms,
                         const double *hs, int64_t ns, int fields, int mutual, double G, int precision, double *out,
                         cudaStream_t st) {
    int W = ((fields & BF_POT) ? 1 : 0) + ((fields & BF_ACC) ? 3 : 0) + ((fields & BF_TID) ? 9 : 0);
    if (nt <= 0) return TG_OK;
    if (mutual) TG_TRY(dispatch_bf<true>(fields, precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st));
    else TG_TRY(dispatch_bf<false>(fields, precision, pt, ht, nt, ps, ms, hs, ns, G, out, W, st));
    TG_CUDA(cudaGetLastError());
    return TG_OK;
}

}  // namespace tg
