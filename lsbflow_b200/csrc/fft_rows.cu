// FP64 row transforms between y-intermediate rows (kx modes) and physical rows (horfft,
// src/horfft.f90:61-150) as the two-step split N = V T of a row's N = nx / 2 complex values: T lanes
// of a warp hold a row, V values each, run V-point register DFTs, exchange through shared memory
// (pitch T + 1: conflict-free) and run T-point DFTs, whose outputs are T-lane runs of the row.  No
// block barrier; global rows are read and written directly.  The lane networks of fft_warp.cu move
// every value log2 T times by shuffles with a select each, which bounds them by issue; here the
// latency of the loads and of the one exchange bounds, with 20 to 28 warps on an SM.
// Measured, mean launch of the SGS models' fields, networks -> split, in us (inverse; forward), at
// nx x ny x nz points: N = 48 (96 x 40 x 64) 12.4 -> 9.6; 10.7 -> 9.7.  64 (128 x 32 x 97)
// 19.6 -> 12.7; 22.7 -> 16.8.  72 (144 x 32 x 96) 25.4 -> 23.0; 14.4 -> 12.6.  96 (192 x 48 x 81)
// 34.3 -> 29.8; 31.1 -> 27.7.  112 (224 x 32 x 64) 22.6 -> 19.5; 14.1 -> 11.3.  128 (256 x 64 x 129)
// 58.7 -> 52.5; 31.2 -> 28.7.  144 (288 x 32 x 64) 35.9 -> 28.4; 21.9 -> 15.8.
#include "lsb_fftdev.cuh"
#include "lsb_internal.cuh"

namespace lsb {
namespace {

constexpr int NW = 4;  // warps per block

__host__ __device__ constexpr int row_pitch(int V, int T) { return V * (T + 1); }
// blocks per SM: 96, 80, 72 registers a thread (6 to 8 values on 16 lanes in 72 spill: 33.9, 54.8 us
// instead of 29.8, 52.5 for the inverse rows of 96 and 128)
__host__ __device__ constexpr int row_blocks(int V, int T) { return V > 8 ? 5 : T == 16 ? 6 : 7; }

template <int V, int T, int SIGN>
__device__ __forceinline__ void split_fft(double2 (&v)[V], double2 (&x)[(V + T - 1) / T][T], int t, double2* S,
                                          const double2* __restrict__ tw) {
    dft_reg<V, SIGN>(v);
#pragma unroll
    for (int k = 0; k < V; ++k) {
        if (k > 0) {
            double2 w = __ldg(&tw[t * k]);
            if (SIGN > 0) w.y = -w.y;
            v[k] = cmul(v[k], w);
        }
        S[k * (T + 1) + t] = v[k];
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < (V + T - 1) / T; ++u) {
        const int k = t + T * u;
        if (V % T != 0 && k >= V) break;
#pragma unroll
        for (int q = 0; q < T; ++q) x[u][q] = S[k * (T + 1) + q];
        dft_reg<T, SIGN>(x[u]);  // x[u][q]: value k + V q of the result
    }
}

template <int V, int T>
__global__ void __launch_bounds__(32 * NW, row_blocks(V, T)) k_row_c2r_v(RowJobList jobs, RowArgs a, unsigned nunits) {
    constexpr int N = V * T, LPW = 32 / T, U = (V + T - 1) / T;
    extern __shared__ __align__(16) double2 sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane / T, t = lane - g * T;
    double2* S = sm + (warp * LPW + g) * row_pitch(V, T);
    const unsigned nrows = (unsigned)(a.nyl * a.nzp);
    const unsigned u0 = (blockIdx.x * NW + warp) * LPW;
    if (u0 >= nunits) return;
    const bool act = u0 + g < nunits;  // a group past the last row repeats it, unstored
    const unsigned unit = act ? u0 + g : nunits - 1;
    const int jb = (int)(unit / nrows);
    const unsigned row = unit - jb * nrows;
    const RowIO& job = jobs.j[jb];
    const int K = a.kxc;
    const double2* src = reinterpret_cast<const double2*>(job.yin) + (size_t)row * K;
    const double2 zero = make_double2(0.0, 0.0);
    double2 v[V];
#pragma unroll
    for (int n = 0; n < V; ++n) {
        const int k = t + T * n;
        double2 xa = (k < K) ? src[k] : zero, xb = (N - k < K) ? src[N - k] : zero;
        if (job.mode == YM_IKX) {
            const double ka = (k < K) ? __ldg(&a.wavx[2 * k]) : 0.0, kb = (N - k < K) ? __ldg(&a.wavx[2 * (N - k)]) : 0.0;
            xa = make_double2(-ka * xa.y, ka * xa.x);
            xb = make_double2(-kb * xb.y, kb * xb.x);
        }
        if (k == 0) xa.y = 0.0;  // FFTW c2r ignores Im of the DC input
        xb = cconj(xb);
        const double2 e = cadd(xa, xb);
        const double2 o = cmul(csub(xa, xb), cconj(__ldg(&a.rp.twr[k])));
        v[n] = make_double2(e.x - o.y, e.y + o.x);
    }
    double2 x[U][T];
    split_fft<V, T, +1>(v, x, t, S, a.rp.half.tw);
    const double m = (job.mean != nullptr && job.add_mean != 0.0) ? job.mean[row / a.nyl] * job.add_mean : 0.0;
    double2* out = reinterpret_cast<double2*>(job.out + (long long)row * a.row_pitch);
    if (!act) return;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = t + T * u;
        if (V % T != 0 && k >= V) break;
#pragma unroll
        for (int q = 0; q < T; ++q)
            out[k + V * q] = make_double2(job.scale * x[u][q].x + m, job.scale * x[u][q].y + m);
    }
}

template <int V, int T>
__global__ void __launch_bounds__(32 * NW, row_blocks(V, T)) k_row_r2c_v(RowJobList jobs, RowArgs a, unsigned nunits) {
    constexpr int N = V * T, LPW = 32 / T, U = (V + T - 1) / T;
    extern __shared__ __align__(16) double2 sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane / T, t = lane - g * T;
    double2* S = sm + (warp * LPW + g) * row_pitch(V, T);
    const unsigned nrows = (unsigned)(a.nyl * a.nzp);
    const unsigned u0 = (blockIdx.x * NW + warp) * LPW;
    if (u0 >= nunits) return;
    const bool act = u0 + g < nunits;
    const unsigned unit = act ? u0 + g : nunits - 1;
    const int jb = (int)(unit / nrows);
    const unsigned row = unit - jb * nrows;
    const RowIO& job = jobs.j[jb];
    const double2* in = reinterpret_cast<const double2*>(job.yin + (long long)row * a.row_pitch);
    double2 v[V];
#pragma unroll
    for (int n = 0; n < V; ++n) v[n] = in[t + T * n];
    if (job.lam != nullptr) {  // fringe forcing lambda(x) (m - q) on the fly
        const double m = (job.mean != nullptr && job.add_mean != 0.0) ? job.mean[row / a.nyl] * job.add_mean : 0.0;
#pragma unroll
        for (int n = 0; n < V; ++n) {
            const double2 l = __ldg(reinterpret_cast<const double2*>(job.lam) + t + T * n);
            v[n] = make_double2(l.x * (m - v[n].x), l.y * (m - v[n].y));
        }
    }
    double2 x[U][T];
    split_fft<V, T, -1>(v, x, t, S, a.rp.half.tw);
    __syncwarp();  // the exchange has been read: the row goes there in natural order
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k = t + T * u;
        if (V % T != 0 && k >= V) break;
#pragma unroll
        for (int q = 0; q < T; ++q) S[k + V * q] = x[u][q];
    }
    __syncwarp();
    if (!act) return;
    const int K = a.kxc;
    double2* out = reinterpret_cast<double2*>(job.out) + (size_t)row * K;
#pragma unroll
    for (int n = 0; n < V; ++n) {
        const int k = t + T * n;
        if (k < K) {
            const double2 za = S[k], zb = cconj(S[k == 0 ? 0 : N - k]);
            const double2 e = make_double2(0.5 * (za.x + zb.x), 0.5 * (za.y + zb.y));
            const double2 o = make_double2(0.5 * (za.x - zb.x), 0.5 * (za.y - zb.y));
            const double2 w = cmul(__ldg(&a.rp.twr[k]), o);
            out[k] = make_double2(e.x + w.y, e.y - w.x);
        }
    }
}

template <int V, int T>
bool launch(const RowJobList& jobs, const RowArgs& a, cudaStream_t s, bool c2r) {
    const long long n = (long long)jobs.n * a.nyl * a.nzp;
    const long long blocks = (n + NW * (32 / T) - 1) / (NW * (32 / T));
    if (n >= (1LL << 31)) return false;
    const size_t smem = (size_t)NW * (32 / T) * row_pitch(V, T) * sizeof(double2);
    const void* kern = c2r ? (const void*)k_row_c2r_v<V, T> : (const void*)k_row_r2c_v<V, T>;
    if (!allow_smem(kern, smem)) return false;
    lsb::note_launch();
    if (c2r) k_row_c2r_v<V, T><<<(int)blocks, 32 * NW, smem, s>>>(jobs, a, (unsigned)n);
    else k_row_r2c_v<V, T><<<(int)blocks, 32 * NW, smem, s>>>(jobs, a, (unsigned)n);
    return true;
}

}  // namespace

// The lengths are those with V = 6 to 9 on 8 or 16 lanes.  Outside, the networks were as good or
// better (us, networks against split, inverse; forward): 32 = 8 x 4 3.2 / 3.8; 3.2 / 4.3.
// 80 = 10 x 8 16.1 / 18.8; 10.5 / 12.2.  96 = 12 x 8 34.3 / 35.9; 31.1 / 33.5.  128 = 16 x 8
// 58.7 / 59.8; 31.2 / 33.5.  160 = 10 x 16 16.7 / 19.0; 10.9 / 12.7.  256 = 16 x 16 111 / 115;
// 57.9 / 59.0: from 10 values a lane on the registers leave too few warps, and 4-lane rows are too short.
bool launch_row_split(const RowJobList& jobs, const RowArgs& a, cudaStream_t s, bool c2r) {
    if (a.f32 || !a.split) return false;
    switch (a.nxl / 2) {
#define LSB_RS(v, t) \
    case (v) * (t): return launch<v, t>(jobs, a, s, c2r);
        LSB_RS(6, 8) LSB_RS(7, 8) LSB_RS(8, 8) LSB_RS(9, 8)
        LSB_RS(6, 16) LSB_RS(7, 16) LSB_RS(8, 16) LSB_RS(9, 16)
#undef LSB_RS
        default: return false;
    }
}

}  // namespace lsb
