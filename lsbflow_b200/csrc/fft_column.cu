// FP64 spanwise passes (horfft, src/horfft.f90:61-150, and the padded passes of
// dealiasing_2d_fftw, src/dealiasing.f90:262-447): N = V T values of a kx column are held by T
// threads, V each, in registers.  Threads are laid out with the column fastest, so that a warp
// reads and writes 32 neighbouring columns of a row (512 bytes) straight from and to global memory.
// With T = 1 (N <= 24) a column is one register DFT; above that the transform is the two-step split
// N = V x T: a V-point DFT over the values t + T n of each thread, the twiddles exp(-+2 pi i t k / N),
// one exchange through shared memory (conflict-free: columns are contiguous there too) and T-point
// DFTs.  No input is staged, no value crosses lanes, and the block (T warps) meets one barrier, where
// the tiled pass of fft_warp.cu stages its tile, runs log2 of its lane group's stages of shuffles on
// it and writes it back through shared memory: that pass is bound by instruction issue, this one by
// DRAM, and on small grids by the latency of one round of loads.
#include <stdexcept>

#include "lsb_fftdev.cuh"
#include "lsb_internal.cuh"

namespace lsb {
namespace {

constexpr int CB = 32;  // columns per block: one warp's

// padded row -> input row, or -1 for a row of the zero pad (the inverse of pad_row)
__device__ __forceinline__ int unpad_row_c(int n, int ny, int nyl, int layout) {
    if (layout == 0 || nyl == ny) return n < ny ? n : -1;
    if (n < ny / 2) return n;
    if (n >= nyl - (ny - ny / 2)) return n - (nyl - ny);
    return -1;
}
__device__ __forceinline__ int pad_row_c(int j, int ny, int nyl, int layout) {
    if (layout == 0 || nyl == ny) return j;
    return (j < ny / 2) ? j : j + (nyl - ny);
}

// warps per block: the T warps of 32 columns, or four independent ones
__host__ __device__ constexpr int ycol_warps(int T) { return T == 1 ? 4 : T; }
// blocks per SM that the register budget is held to: more warps beat a few spills (256x64x129, 28
// against 20 warps at V = 8 and 24 against 16 at V = 12: forward passes 89 -> 77 us padded, 75 ->
// 68 us accumulating), except for accumulating jobs of V > 8, which also hold their old values
__host__ __device__ constexpr int ycol_blocks(int V, int T, bool acc) {
    const int w = V <= 8 ? 28 : (V <= 12 && !acc ? 24 : (V <= 16 ? 16 : 12));
    return w / ycol_warps(T) > 0 ? w / ycol_warps(T) : 1;
}

// ACC: some job of a forward launch adds to its output
template <int V, int T, bool INV, bool ACC>
__global__ void __launch_bounds__(32 * ycol_warps(T), ycol_blocks(V, T, ACC))
    k_ycol(YInvJobList ij, YFwdJobList fj, YPassArgs a, unsigned nunits, unsigned nch) {
    constexpr int N = V * T, U = (V + T - 1) / T;  // U: T-point DFTs per thread
    constexpr int SIGN = INV ? +1 : -1;
    extern __shared__ __align__(16) double2 sm[];  // [V][T][CB] (T > 1)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // unit = (z, chunk of 32 columns, job), the job fastest: the fields that share an input (u and
    // du/dy) read it at about the same time
    const unsigned unit = T == 1 ? blockIdx.x * ycol_warps(T) + warp : blockIdx.x;
    if (unit >= nunits) return;  // (uniform over the block for T > 1)
    const unsigned njobs = INV ? ij.n : fj.n;
    const int jb = (int)(unit % njobs);
    const unsigned rest = unit / njobs;
    const int ch = (int)(rest % nch), z = (int)(rest / nch);
    const int c = ch * CB + lane, t = T == 1 ? 0 : warp;
    const bool act = c < a.kxc;
    const int ny = a.ny, h = a.nx / 2;
    const int rows_in = INV ? ny : N, rows_out = INV ? N : ny;
    const double2* in = reinterpret_cast<const double2*>(INV ? ij.j[jb].in : fj.j[jb].in) +
                        (long long)z * rows_in * h + c;
    double2* out = reinterpret_cast<double2*>(INV ? ij.j[jb].out : fj.j[jb].out) + (long long)z * rows_out * h + c;
    const double2 zero = make_double2(0.0, 0.0);

    double2 v[V];
#pragma unroll
    for (int n = 0; n < V; ++n) {
        const int row = INV ? unpad_row_c(t + T * n, ny, N, a.layout) : t + T * n;
        v[n] = (act && row >= 0) ? in[(long long)row * h] : zero;
    }
    if (INV && ij.j[jb].mode != YM_COPY) {
        const bool ikx = ij.j[jb].mode == YM_IKX;
        const double kx = (ikx && act) ? a.wavx[2 * c] : 0.0;
#pragma unroll
        for (int n = 0; n < V; ++n) {
            const int row = unpad_row_c(t + T * n, ny, N, a.layout);
            const double k = ikx ? kx : (row >= 0 ? a.wavy[row] : 0.0);
            v[n] = make_double2(-k * v[n].y, k * v[n].x);
        }
    }
    dft_reg<V, SIGN>(v);

    // output row o (of N), from this thread's unit
    const double alpha = INV ? 1.0 : fj.j[jb].alpha, beta = ACC ? fj.j[jb].beta : 0.0;
    const bool sym = !INV && fj.j[jb].sym && ch == 0;  // the kx = 0 column of this block is symmetrised
    auto store = [&](int o, double2 x, double2 old) {
        if (INV) {
            out[(long long)o * h] = x;
        } else {
            const int j = unpad_row_c(o, ny, N, a.layout);
            x.x *= a.scale;
            x.y *= a.scale;
            out[(long long)j * h] = (ACC && beta != 0.0) ? make_double2(fma(alpha, x.x, beta * old.x), fma(alpha, x.y, beta * old.y))
                                                          : make_double2(alpha * x.x, alpha * x.y);
        }
    };
    auto kept = [&](int o) { return act && (INV || unpad_row_c(o, ny, N, a.layout) >= 0); };
    const double2* prev = ACC ? reinterpret_cast<const double2*>(fj.j[jb].prev) + (long long)z * rows_out * h + c : nullptr;
    auto previous = [&](int o) {
        return (ACC && beta != 0.0 && kept(o)) ? prev[(long long)unpad_row_c(o, ny, N, a.layout) * h] : zero;
    };
    auto mirror = [&](int o) {  // the row that the Hermitian symmetrisation pairs with o
        return pad_row_c((ny - unpad_row_c(o, ny, N, a.layout)) % ny, ny, N, a.layout);
    };
    if constexpr (T == 1) {
        if (sym && c == 0) {
            double2 w[V];
#pragma unroll
            for (int o = 0; o < V; ++o) w[o] = v[o];
#pragma unroll
            for (int o = 0; o < V; ++o)
                if (kept(o)) {
                    const double2 m = w[mirror(o)];
                    v[o] = make_double2(0.5 * (v[o].x + m.x), 0.5 * (v[o].y - m.y));
                }
        }
        if (ACC && beta != 0.0) {
            double2 old[V];
#pragma unroll
            for (int o = 0; o < V; ++o) old[o] = previous(o);
#pragma unroll
            for (int o = 0; o < V; ++o)
                if (kept(o)) store(o, v[o], old[o]);
        } else {
#pragma unroll
            for (int o = 0; o < V; ++o)
                if (kept(o)) store(o, v[o], zero);
        }
    } else {
#pragma unroll
        for (int k = 0; k < V; ++k) {
            if (k > 0) {
                double2 w = __ldg(&a.plan.tw[t * k]);  // the same for the whole warp
                if (SIGN > 0) w.y = -w.y;
                v[k] = cmul(v[k], w);
            }
            sm[(k * T + t) * CB + lane] = v[k];
        }
        // thread t takes the units k = t + T u: rows k + V q, q < T
        double2 old[U][ACC ? T : 1];
        if (ACC && beta != 0.0) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < T; ++q)
                    if (V % T == 0 || t + T * u < V) old[u][ACC ? q : 0] = previous(t + T * u + V * q);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = t + T * u;
            if (V % T != 0 && k >= V) break;
            double2 x[T];
#pragma unroll
            for (int q = 0; q < T; ++q) x[q] = sm[(k * T + q) * CB + lane];
            dft_reg<T, SIGN>(x);
            if (sym) {  // back to shared memory, where the mirrored rows are read after a barrier
#pragma unroll
                for (int q = 0; q < T; ++q) sm[(k * T + q) * CB + lane] = x[q];
            } else {
#pragma unroll
                for (int q = 0; q < T; ++q)
                    if (kept(k + V * q)) store(k + V * q, x[q], (ACC && beta != 0.0) ? old[u][ACC ? q : 0] : zero);
            }
        }
        if (!INV && sym) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = t + T * u;
                if (V % T != 0 && k >= V) break;
#pragma unroll
                for (int q = 0; q < T; ++q) {
                    const int o = k + V * q;
                    if (!kept(o)) continue;
                    double2 x = sm[(k * T + q) * CB + lane];
                    if (c == 0) {
                        const int m = mirror(o);
                        const double2 y = sm[((m % V) * T + m / V) * CB];
                        x = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
                    }
                    store(o, x, (ACC && beta != 0.0) ? old[u][ACC ? q : 0] : zero);
                }
            }
        }
    }
}

template <int V, int T, bool INV>
bool launch(const YInvJobList& ij, const YFwdJobList& fj, const YPassArgs& a, cudaStream_t s) {
    const unsigned nch = (a.kxc + CB - 1) / CB;
    const unsigned nunits = (unsigned)((INV ? ij.n : fj.n) * a.nzp) * nch;
    constexpr int W = ycol_warps(T);
    const unsigned blocks = T == 1 ? (nunits + W - 1) / W : nunits;
    const size_t smem = T == 1 ? 0 : (size_t)V * T * CB * sizeof(double2);
    auto go = [&](auto kern) {
        if (!allow_smem((const void*)kern, smem)) return false;
        lsb::note_launch();
        kern<<<blocks, 32 * W, smem, s>>>(ij, fj, a, nunits, nch);
        return true;
    };
    if constexpr (INV) {
        return go(k_ycol<V, T, true, false>);
    } else {
        bool acc = false;
        for (int i = 0; i < fj.n; ++i) acc = acc || fj.j[i].beta != 0.0;
        return acc ? go(k_ycol<V, T, false, true>) : go(k_ycol<V, T, false, false>);
    }
}

template <bool INV>
bool dispatch(const YInvJobList& ij, const YFwdJobList& fj, const YPassArgs& a, cudaStream_t s) {
    if (a.f32 || !a.column) return false;
    // The split: few values per thread make many warps, few threads make few T-point steps; the
    // padded inverse, whose row tests cost registers, is faster with fewer values than the forward
    // pass (48: 9.2 us at 8 x 6, 13.8 at 12 x 4 inverse, 13.4 and 10.7 forward, 128x32x65).
    switch (a.nyl) {
#define LSB_YC(v, t) \
    case (v) * (t): return launch<v, t, INV>(ij, fj, a, s);
#define LSB_YC2(v, t, w, u) \
    case (v) * (t): static_assert((v) * (t) == (w) * (u), ""); return launch<INV ? v : w, INV ? t : u, INV>(ij, fj, a, s);
        LSB_YC(2, 1) LSB_YC(3, 1) LSB_YC(4, 1) LSB_YC(5, 1) LSB_YC(6, 1) LSB_YC(7, 1) LSB_YC(8, 1) LSB_YC(9, 1)
        LSB_YC(10, 1) LSB_YC(12, 1) LSB_YC(7, 2) LSB_YC(5, 3) LSB_YC(4, 4) LSB_YC(9, 2) LSB_YC(5, 4) LSB_YC(8, 3)
        LSB_YC(7, 4) LSB_YC(10, 3) LSB_YC(8, 4) LSB_YC(9, 4) LSB_YC2(8, 5, 10, 4) LSB_YC(7, 6) LSB_YC2(8, 6, 12, 4)
        LSB_YC(9, 6) LSB_YC(8, 7) LSB_YC2(10, 6, 12, 5) LSB_YC(8, 8) LSB_YC2(9, 8, 12, 6) LSB_YC(10, 8)
        LSB_YC(12, 7) LSB_YC(10, 9) LSB_YC2(8, 12, 12, 8) LSB_YC(12, 9) LSB_YC(14, 8) LSB_YC2(10, 12, 12, 10)
        LSB_YC(16, 8) LSB_YC(12, 12) LSB_YC(16, 12) LSB_YC(7, 3) LSB_YC(5, 5) LSB_YC(9, 3) LSB_YC(7, 5) LSB_YC(9, 5)
        LSB_YC(9, 7)
#undef LSB_YC
#undef LSB_YC2
        default: return false;
    }
}

}  // namespace

bool launch_yinv_column(const YInvJobList& jobs, const YPassArgs& a, cudaStream_t s) {
    return dispatch<true>(jobs, YFwdJobList{}, a, s);
}
bool launch_yfwd_column(const YFwdJobList& jobs, const YPassArgs& a, cudaStream_t s) {
    return dispatch<false>(YInvJobList{}, jobs, a, s);
}

}  // namespace lsb
