// The fused nonlinear-product rows (nlterm_skewsym, src/navierstokes.f90:725-769) in FP64 for rows
// of 384 complex values, the padded rows of 512-point grids: a warp owns a (z, y) row, 12 values per
// lane, and runs its 12 c2r, the skew-symmetric products and 9 r2c, as k_row_nl_r (fft_warp.cu) does
// with the exchange network.  What differs is the cross-lane part of a transform.  There it is five
// radix-2 stages, each a shuffle and selects per value and four FP64 instructions; here one radix-2
// stage by shuffles and two radix-4 steps whose values move through shared memory (4 x 4 transposes
// between four lanes, 16-byte accesses without bank conflicts): two thirds of the instructions.
// Both run at 7 to 8 warps per SM, set by the 12 values a lane keeps of three velocity rows, and
// are bound by latency there, so that nothing in a row's chain waits for global memory here: the
// next c2r's input row is copied to shared memory behind the current transform, and the twiddles of
// the first step and of the real-to-complex split sit there as well (without that the radix-4 form
// gained nothing, 926 us).  96 x 129 rows: 907 -> 734 us, 512x64x129 step 3612 -> 3455 us.  The
// same scheme on 192 values (16 lanes, two rows a warp) measured 317 against 324 us, on 96 (8 lanes)
// 51 against 46: those lengths keep the exchange network at 12 warps per SM.
#include "lsb_fftdev.cuh"
#include "lsb_internal.cuh"

namespace lsb {
namespace {

constexpr int R = 12, G = 32, N = R * G;
constexpr int NW = 7;  // warps per block, one block per SM

// index of value i = 4 m + j of lane g in the row, after sfft / before sfft_dit
__device__ __forceinline__ int sslot(int g, int i) {
    const int col = ((g >> 2) & 3) + 4 * (i >> 2), par = col >= 6 ? 1 : 0;
    return col - 6 * par + 6 * (g >> 4) + R * (2 * ((g & 3) + 4 * (i & 3)) + par);
}

template <int SIGN>
__device__ __forceinline__ double2 twid(const double2* __restrict__ tw, int i) {
    double2 w = __ldg(&tw[i]);
    if (SIGN > 0) w.y = -w.y;
    return w;
}

template <int SIGN>
__device__ __forceinline__ void dft4(double2 (&v)[R], int m, const double2 (&x)[4]) {
    double2 u[4] = {x[0], x[1], x[2], x[3]};
    dft_reg<4, SIGN>(u);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[4 * m + j] = u[j];
}

__device__ __forceinline__ double2 shfl_xor2(double2 x, int h) {
    return make_double2(__shfl_xor_sync(0xffffffffu, x.x, h), __shfl_xor_sync(0xffffffffu, x.y, h));
}

// DFT of a row from natural order (lane g, register r: x[g + G r]) to the slots above.  B: the
// exchange buffer of the lane's half warp (12 rows of 20);
// T: exp(-2 pi i g k / N) as [k - 1][g], in shared memory
template <int SIGN>
__device__ __forceinline__ void sfft(double2 (&v)[R], int g, double2* B, const double2* T,
                                     const double2* __restrict__ tw) {
    dft_reg<R, SIGN>(v);
#pragma unroll
    for (int k = 1; k < R; ++k) {
        double2 w = T[(k - 1) * G + g];
        if (SIGN > 0) w.y = -w.y;
        v[k] = cmul(v[k], w);
    }
    // radix 2 over the lanes g, g ^ G/2: the lower one takes columns 0..5, the upper 6..11
    const bool up = (g & (G / 2)) != 0;
    const double2 w2 = twid<SIGN>(tw, (N / G) * (g & (G / 2 - 1)));
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 own = up ? v[6 + i] : v[i];
        const double2 r = shfl_xor2(up ? v[i] : v[6 + i], G / 2);
        const double2 lo = up ? r : own, hi = up ? own : r;
        v[i] = cadd(lo, hi);
        v[6 + i] = cmul(csub(lo, hi), w2);
    }
    __syncwarp();
    const int l = g & 15, a = l & 3, b = l >> 2;
    double2 w[4];
#pragma unroll
    for (int j = 1; j < 4; ++j) w[j] = twid<SIGN>(tw, (N / 16) * a * j);
#pragma unroll
    for (int c = 0; c < R; ++c) B[c * 20 + l] = v[c];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        double2 x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = B[(b + 4 * m) * 20 + a + 4 * q];
        dft4<SIGN>(v, m, x);
#pragma unroll
        for (int j = 1; j < 4; ++j) v[4 * m + j] = cmul(v[4 * m + j], w[j]);
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) B[(b + 4 * m) * 20 + a * 5 + j] = v[4 * m + j];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        double2 x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = B[(b + 4 * m) * 20 + q * 5 + a];
        dft4<SIGN>(v, m, x);
    }
}

// the transpose: from the slots to natural order
template <int SIGN>
__device__ __forceinline__ void sfft_dit(double2 (&v)[R], int g, double2* B, const double2* T,
                                         const double2* __restrict__ tw) {
    const int l = g & 15, a = l & 3, b = l >> 2;
    double2 w[4];
#pragma unroll
    for (int j = 1; j < 4; ++j) w[j] = twid<SIGN>(tw, (N / 16) * a * j);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const double2 x[4] = {v[4 * m], v[4 * m + 1], v[4 * m + 2], v[4 * m + 3]};
        dft4<SIGN>(v, m, x);
#pragma unroll
        for (int j = 1; j < 4; ++j) v[4 * m + j] = cmul(v[4 * m + j], w[j]);
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) B[(b + 4 * m) * 20 + a * 5 + j] = v[4 * m + j];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        double2 x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = B[(b + 4 * m) * 20 + q * 5 + a];
        dft4<SIGN>(v, m, x);
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) B[(b + 4 * m) * 20 + a + 4 * j] = v[4 * m + j];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < R; ++c) v[c] = B[c * 20 + l];
    const bool up = (g & (G / 2)) != 0;
    const double2 w2 = twid<SIGN>(tw, (N / G) * (g & (G / 2 - 1)));
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double2 o = cmul(v[6 + i], w2);
        const double2 s = cadd(v[i], o), d = csub(v[i], o);
        const double2 r = shfl_xor2(up ? s : d, G / 2);
        v[i] = up ? r : s;
        v[6 + i] = up ? d : r;
    }
#pragma unroll
    for (int k = 1; k < R; ++k) {
        double2 w = T[(k - 1) * G + g];
        if (SIGN > 0) w.y = -w.y;
        v[k] = cmul(v[k], w);
    }
    dft_reg<R, SIGN>(v);
}

constexpr int kExch = 2 * R * 20;
// per warp: the three velocity rows (lane-private), the exchange buffer; the staged input row
// follows
constexpr int kWarp = 3 * R * 32 + kExch;
inline size_t row_smem(int K) {
    return (size_t)(NW * (kWarp + K) + (R - 1) * G + N) * sizeof(double2);
}

__device__ __forceinline__ void cpa16s(void* d, const void* g) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g));
}

__global__ void __launch_bounds__(32 * NW, 1) k_row_nl_s(NlRowArgs a) {
    const RowArgs& r = a.r;
    const int K = r.kxc;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane;
    const int nitems = r.nyl * r.nzp;
    const int step = gridDim.x * NW;
    extern __shared__ __align__(16) double2 sm[];
    double2* T = sm;                       // [R - 1][G]
    double2* twr = T + (R - 1) * G;        // [N]
    double2* us = twr + N + warp * (kWarp + K);  // u, v, w of the warp's row, lane-private
    double2* B = us + 3 * R * 32 + (lane >> 4) * (R * 20);
    double2* st = us + kWarp;              // the staged input row
    auto U = [&](int l, int i) -> double2& { return us[(l * R + i) * 32 + lane]; };
    const double2* __restrict__ tw = r.rp.half.tw;
    for (int i = threadIdx.x; i < (R - 1) * G; i += 32 * NW) T[i] = tw[(i % G) * (i / G + 1)];
    for (int i = threadIdx.x; i < N; i += 32 * NW) twr[i] = r.rp.twr[i];
    __syncthreads();
    const double2 zero = make_double2(0.0, 0.0);
    const int mir = (G - g) & (G - 1);     // the lane of Z[N - k]
    auto input = [&](int op) {  // the row set of c2r op 0..2, 9..11, 13..15, 17..19
        const int cl = (op - 9) >> 2, ct = (op - 9) & 3;
        return (op < 3) ? a.U[op] : (ct == 0 ? a.U[cl] : (ct == 1 ? a.DY[cl] : a.DZ[cl]));
    };
    auto stage = [&](const double* f, int row) {
        const double2* src = reinterpret_cast<const double2*>(f) + (long long)row * K;
        for (int k = g; k < K; k += G) cpa16s(st + k, src + k);
    };
    int row = blockIdx.x * NW + warp;
    if (row < nitems) stage(a.U[0], row);
    for (; row < nitems; row += step) {
        const int z = row / r.nyl;
        const long long off = (long long)row * 2 * K;
        const double ub = a.ubar[z], ubp = a.ubarp[z];
        double2 conv[R];  // -0.5 u_m d_m u_l of the current component
#pragma unroll
        for (int i = 0; i < R; ++i) conv[i] = zero;
        // the ops of k_row_nl_r: 0..2 c2r of u_l; 3..8 r2c of the fluxes; 9..20 per component the
        // c2r of its three gradients and the r2c of the convective sum
#pragma unroll 1
        for (int op = 0; op < 21; ++op) {
            const int cl = (op - 9) >> 2, ct = (op - 9) & 3;
            double2 v[R];
            if (op < 3 || (op >= 9 && ct < 3)) {
                const bool ikx = op >= 9 && ct == 0;
                asm volatile("cp.async.wait_all;\n" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    const int n = g + G * rr;
                    double2 xa = zero, xb = zero;
                    if (n < K) xa = st[n];
                    if (N - n < K) xb = st[N - n];
                    if (ikx) {
                        const double ka = (n < K) ? __ldg(&r.wavx[2 * n]) : 0.0;
                        const double kb = (N - n < K) ? __ldg(&r.wavx[2 * (N - n)]) : 0.0;
                        xa = make_double2(-ka * xa.y, ka * xa.x);
                        xb = make_double2(-kb * xb.y, kb * xb.x);
                    }
                    if (n == 0) xa.y = 0.0;  // FFTW c2r ignores Im of the DC input
                    xb = cconj(xb);
                    const double2 e = cadd(xa, xb);
                    const double2 o = cmul(csub(xa, xb), cconj(twr[n]));
                    v[rr] = make_double2(e.x - o.y, e.y + o.x);
                }
                __syncwarp();  // the staged row has been read
                const int nop = op == 2 ? 9 : ((ct == 2 && op >= 9) ? op + 2 : op + 1);
                if (nop < 20) stage(input(nop), row);
                else if (row + step < nitems) stage(a.U[0], row + step);
                sfft<+1>(v, g, B, T, tw);
                if (op < 3) {
                    const double add = (op == 0) ? ub : 0.0;
#pragma unroll
                    for (int i = 0; i < R; ++i) U(op, i) = make_double2(v[i].x + add, v[i].y + add);
                } else {
                    const double dzb = (ct == 2 && cl == 0) ? ubp : 0.0;
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const double2 um = U(ct, i);
                        const double2 c = (ct == 0) ? zero : conv[i];
                        conv[i] = make_double2(c.x - 0.5 * (um.x * (v[i].x + dzb)), c.y - 0.5 * (um.y * (v[i].y + dzb)));
                    }
                }
            } else {
                double* dst;
                if (op < 9) {
                    const int p = op - 3;
                    const int l = (p < 3) ? 0 : (p < 5 ? 1 : 2);
                    const int m = (p < 3) ? p : (p < 5 ? p - 2 : 2);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const double2 ul = U(l, i), um = U(m, i);
                        v[i] = make_double2(0.5 * (ul.x * um.x), 0.5 * (ul.y * um.y));
                    }
                    dst = a.H[p];
                } else {
                    const double ut = (cl == 0) ? ub : 0.0;
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        double2 c = conv[i];
                        if (a.lamx != nullptr) {
                            const int x = 2 * sslot(g, i);  // physical x of the pair in register i
                            const double lx0 = __ldg(&a.lamx[x]), lx1 = __ldg(&a.lamx[x + 1]);
                            const double2 ul = U(cl, i);
                            c.x = c.x + lx0 * (ut - ul.x);
                            c.y = c.y + lx1 * (ut - ul.y);
                        }
                        v[i] = c;
                    }
                    dst = a.N[cl];
                }
                sfft_dit<-1>(v, g, B, T, tw);
                // Z[N-k] for k = g + G rr: lane (G-g) register R-1-rr (g > 0), or lane 0 register R-rr
                double2* o2 = reinterpret_cast<double2*>(dst + off);
#pragma unroll
                for (int rr = 0; rr < R; ++rr) {
                    double2 zb;
                    zb.x = __shfl_sync(0xffffffffu, v[R - 1 - rr].x, mir);
                    zb.y = __shfl_sync(0xffffffffu, v[R - 1 - rr].y, mir);
                    if (g == 0) zb = v[rr == 0 ? 0 : R - rr];
                    const int k = g + G * rr;
                    if (k < K) {
                        const double2 za = v[rr];
                        zb = cconj(zb);
                        const double2 e = make_double2(0.5 * (za.x + zb.x), 0.5 * (za.y + zb.y));
                        const double2 o = make_double2(0.5 * (za.x - zb.x), 0.5 * (za.y - zb.y));
                        const double2 t = cmul(twr[k], o);
                        o2[k] = make_double2(e.x + t.y, e.y - t.x);
                    }
                }
            }
        }
    }
}

bool launch(const NlRowArgs& a, cudaStream_t s) {
    const size_t sm = row_smem(a.r.kxc);
    if (!allow_smem((const void*)k_row_nl_s, sm)) return false;
    const long long rows = (long long)a.r.nyl * a.r.nzp;
    const long long need = (rows + NW - 1) / NW;
    const long long blocks = need < sm_count() ? need : sm_count();
    lsb::note_launch();
    k_row_nl_s<<<(int)blocks, 32 * NW, sm, s>>>(a);
    return true;
}

}  // namespace

bool launch_row_nl_twelve(const NlRowArgs& a, cudaStream_t s) {
    if (a.r.f32) return false;
    return a.r.nxl == 2 * N && launch(a, s);
}

}  // namespace lsb
