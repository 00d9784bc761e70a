// FP64 z contractions on the tensor cores: out = A . in over every (kx, ky) column.
//
// These are the Chebyshev derivatives dfdz / d2fdz2 (src/derivatives.f90:112-188, the
// DCT-I path of src/chebyshev.f90:204-270 written as its dense matrix) and the two
// eigenbasis products of solve_helmholtz (src/helmholtz.f90:130-208), with the
// lifting-function prologue / epilogue of solve_nhom_helmholtz (src/helmholtz.f90:
// 324-353) and the Poisson right-hand side of navierstokes_update (src/navierstokes.f90:
// 1411-1464) fused in.  Accumulating into a field that the epilogue must read back costs
// the read's full latency at the end of every block, so the step stores plain products
// (dz of h_l3, Dw for the pressure) and adds them in its elementwise passes.
//
// tcgen05 has no FP64 kind, so the FP64 form uses the FP64 tensor-core MMA
// (mma.sync m16n8k8 f64: 1024 FMAs per instruction).  One CTA owns all Mp rows of a block
// of 32..64 columns (8 per warp), A and B staged through shared memory in k-chunks of 16 (a
// 3-stage ring) or 32 (a double buffer) with conflict-free strides.
#include <type_traits>

#include "lsb_internal.cuh"

namespace lsb {

constexpr int LDA_S = 20;  // doubles; 8r mod 32 distinct for r = 0..3 -> no bank conflicts (36 for
                           // the 32-column chunks: the same residues)

// D (16x8) += A (16x8) B (8x8).  Fragments (g = lane / 4, t = lane % 4): a = A[g][t],
// A[g+8][t], A[g][t+4], A[g+8][t+4]; b = B[t][g], B[t+4][g]; c = D[g][2t], D[g][2t+1],
// D[g+8][2t], D[g+8][2t+1]
__device__ __forceinline__ void dmma16(double (&c)[4], double a0, double a1, double a2, double a3, double b0,
                                       double b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

__device__ __forceinline__ double w2_of(const GemmArgs& g, long long c) {
    // c < C = nx * ny < 2^31 (checked at create): 32-bit division
    const int i = (int)((unsigned)c % (unsigned)g.nx);
    const int j = (int)((unsigned)c / (unsigned)g.nx);
    const double wx = g.wavx[i], wy = g.wavy[j];
    return wx * wx + wy * wy;
}

__device__ __forceinline__ void cp_async16(void* smem_ptr, const void* gptr, int src_bytes) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem_ptr);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gptr), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// The epilogue of a thread's NTL accumulator tiles (row tiles t0, t0 + 1, .. of the output,
// columns cb and cb + 1 of field f) below row rend; erow: the row factors of the NTL tiles
// ([2][er], lam or hb and ht)
template <int NTL>
__device__ __forceinline__ void gemm_epilogue(const GemmArgs& g, int f, const double (&acc)[NTL][4], int t0,
                                              long long cb, int gq, const double* bcb, const double* bct,
                                              const double* erow, int er, int rend) {
    double* __restrict__ out = (f < 4 && g.outf[f]) ? g.outf[f] : g.out + f * g.out_fstride;
    const double* __restrict__ aux = g.aux ? g.aux + f * g.out_fstride : nullptr;
    // per column of this thread: k^2 for the epilogues that need it, the boundary planes
    double ew2[2] = {0.0, 0.0}, eb[2] = {0.0, 0.0}, et[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        if (cb + e >= g.C) continue;
        if (g.epi == EPI_HELM_SCALE || g.epi == EPI_POISSON_RHS) ew2[e] = w2_of(g, cb + e);
        if (g.epi == EPI_LIFT_ADD && bcb != nullptr) {
            eb[e] = bcb[cb + e];
            et[e] = bct[cb + e];
        }
    }
    // one unrolled store loop per epilogue kind (the kind is uniform over the launch)
    auto epilogue = [&](auto kind) {
        constexpr int E = decltype(kind)::value;
        constexpr bool RD = (E == EPI_AXPBY || E == EPI_POISSON_RHS);
        if constexpr (E == EPI_NLDIV) {
            // the thread's two columns (cb, cb + 1) are the real and imaginary parts of one
            // mode: N_l -= i kx h_l1 + i ky h_l2 + d h_l3/dz (src/navierstokes.f90:789-795),
            // the real part first taking -(-kx Im h_l1), then -(-ky Im h_l2), then Re d h_l3/dz
            if (cb >= g.C) return;
            double* __restrict__ Nl = g.nd_N[f];
            const double* __restrict__ hx = g.nd_hx[f];
            const double* __restrict__ hy = g.nd_hy[f];
            const double wx = g.wavx[(int)((unsigned)cb % (unsigned)g.nx)];
            const double wy = g.wavy[(int)((unsigned)cb / (unsigned)g.nx)];
#pragma unroll
            for (int t = 0; t < NTL; ++t) {
                double2 nv[2], xv[2], yv[2];
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int r = (t0 + t) * 16 + hh * 8 + gq;
                    nv[hh] = xv[hh] = yv[hh] = make_double2(0.0, 0.0);
                    if (r < rend) {
                        const long long o = (long long)(r + g.roff) * g.C + cb;
                        nv[hh] = *reinterpret_cast<const double2*>(Nl + o);
                        xv[hh] = *reinterpret_cast<const double2*>(hx + o);
                        yv[hh] = *reinterpret_cast<const double2*>(hy + o);
                    }
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int r = (t0 + t) * 16 + hh * 8 + gq;
                    if (r >= rend) continue;
                    double nr = nv[hh].x, ni = nv[hh].y;
                    nr = nr - (-wx * xv[hh].y);
                    ni = ni - (wx * xv[hh].x);
                    nr = nr - (-wy * yv[hh].y);
                    ni = ni - (wy * yv[hh].x);
                    nr = nr - acc[t][2 * hh];
                    ni = ni - acc[t][2 * hh + 1];
                    *reinterpret_cast<double2*>(Nl + (long long)(r + g.roff) * g.C + cb) = make_double2(nr, ni);
                }
            }
        } else if constexpr (E == EPI_PRESSURE) {
            // the pressure phi = -(Dw + div)/(k^2 dt bdfv) (0 at k = 0; src/navierstokes.f90:
            // 1466-1476) and the projection u -= dt bdfv dphi/dx, v -= dt bdfv dphi/dy
            // (:1478-1488), for the thread's mode
            if (cb >= g.C) return;
            double* __restrict__ pu = g.pp_u;
            double* __restrict__ pv = g.pp_v;
            double* __restrict__ pp = g.pp_p;
            const double* __restrict__ pdiv = g.pp_div;
            const double wx = g.wavx[(int)((unsigned)cb % (unsigned)g.nx)];
            const double wy = g.wavy[(int)((unsigned)cb / (unsigned)g.nx)];
            const double w2 = wx * wx + wy * wy;
            const double dt = g.pp_dt, bdfv = g.pp_bdfv;
            const double dtb = dt * bdfv;
#pragma unroll
            for (int t = 0; t < NTL; ++t) {
                double2 dv[2], uv[2], vv[2];
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int r = (t0 + t) * 16 + hh * 8 + gq;
                    dv[hh] = uv[hh] = vv[hh] = make_double2(0.0, 0.0);
                    if (r < rend) {
                        const long long o = (long long)(r + g.roff) * g.C + cb;
                        dv[hh] = *reinterpret_cast<const double2*>(pdiv + o);
                        uv[hh] = *reinterpret_cast<const double2*>(pu + o);
                        vv[hh] = *reinterpret_cast<const double2*>(pv + o);
                    }
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int r = (t0 + t) * 16 + hh * 8 + gq;
                    if (r >= rend) continue;
                    const long long o = (long long)(r + g.roff) * g.C + cb;
                    const double pr = (w2 == 0.0) ? 0.0 : -(acc[t][2 * hh] + dv[hh].x) / (w2 * dt * bdfv);
                    const double pi = (w2 == 0.0) ? 0.0 : -(acc[t][2 * hh + 1] + dv[hh].y) / (w2 * dt * bdfv);
                    *reinterpret_cast<double2*>(pp + o) = make_double2(pr, pi);
                    *reinterpret_cast<double2*>(pu + o) =
                        make_double2(uv[hh].x - dtb * (-wx * pi), uv[hh].y - dtb * (wx * pr));
                    *reinterpret_cast<double2*>(pv + o) =
                        make_double2(vv[hh].x - dtb * (-wy * pi), vv[hh].y - dtb * (wy * pr));
                }
            }
        } else {
            // the thread's two columns as 16-byte accesses (C and cb are even: cb < C covers both):
            // 8-byte stores of every second double wrote each sector twice
            if (cb >= g.C) return;
            double* __restrict__ o = out + (long long)(t0 * 16 + gq + g.roff) * g.C + cb;
            const double* __restrict__ ro = (E == EPI_POISSON_RHS) ? aux + (o - out) : o;
            const long long r8 = 8 * g.C;
#pragma unroll
            for (int t = 0; t < NTL; ++t) {
                // the field values this tile's epilogue reads, loaded together before its stores
                double2 old[2];
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    old[hh] = make_double2(0.0, 0.0);
                    if (RD && (E == EPI_POISSON_RHS || g.beta != 0.0) && (t0 + t) * 16 + hh * 8 + gq < rend)
                        old[hh] = *reinterpret_cast<const double2*>(ro + (2 * t + hh) * r8);
                }
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int r = t * 16 + hh * 8 + gq;
                    if (t0 * 16 + r >= rend) continue;
                    double v[2] = {acc[t][2 * hh], acc[t][2 * hh + 1]};
                    const double ov[2] = {old[hh].x, old[hh].y};
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if constexpr (E == EPI_AXPBY) {
                            v[e] = g.alpha * v[e] + (g.beta != 0.0 ? g.beta * ov[e] : 0.0);
                        } else if constexpr (E == EPI_HELM_SCALE) {
                            const double dfac = (-ew2[e]) - g.sigma;
                            v[e] = v[e] / (erow[r] + dfac);
                        } else if constexpr (E == EPI_POISSON_RHS) {
                            v[e] = -v[e] - ew2[e] * ov[e];
                        } else if constexpr (E == EPI_LIFT_ADD) {  // acc + hb*bcb + ht*bct
                            if (bcb != nullptr) v[e] = v[e] + erow[r] * eb[e] + erow[er + r] * et[e];
                        }
                    }
                    *reinterpret_cast<double2*>(o + (2 * t + hh) * r8) = make_double2(v[0], v[1]);
                }
            }
        }
    };
    switch (g.epi) {
        case EPI_STORE: epilogue(std::integral_constant<int, EPI_STORE>{}); break;
        case EPI_AXPBY: epilogue(std::integral_constant<int, EPI_AXPBY>{}); break;
        case EPI_HELM_SCALE: epilogue(std::integral_constant<int, EPI_HELM_SCALE>{}); break;
        case EPI_POISSON_RHS: epilogue(std::integral_constant<int, EPI_POISSON_RHS>{}); break;
        case EPI_NLDIV: epilogue(std::integral_constant<int, EPI_NLDIV>{}); break;
        case EPI_PRESSURE: epilogue(std::integral_constant<int, EPI_PRESSURE>{}); break;
        default: epilogue(std::integral_constant<int, EPI_LIFT_ADD>{}); break;
    }
}

// CTA tile: all Mp rows x 8 * NW columns; warp w owns columns 8w..8w+7 over all MT row
// tiles.  A and B chunks arrive by cp.async through a GSTAGES-deep ring with one barrier per
// chunk; the lifted right-hand side of the non-homogeneous solve is formed from the raw
// input as the B fragments are read (the lane's column is fixed, the row factors sit in
// shared memory), so the lifted contractions stream like the plain ones.
//
// Odd Chebyshev sizes (nzp = 2^n + 1) leave one row and one column past a multiple of 16.
// The row (M = 16 MT + 1) is not a 16-row tile of mostly zeros: each lane accumulates it on
// the FP64 pipe from the B values it already holds (its k subset of its fragment column),
// the four lanes of a column are summed at the end, and the epilogue stores it as one more
// tile.  The column (K = 16 (chunks - 1) + 1, no lift) is not a chunk of mostly zeros: it
// is a rank-1 update acc += A[:, K-1] B[K-1, :] after the last chunk.  Both belong to the
// EDGE instantiations (M = 16 MT + 1); the others compile without them.
constexpr int GSTAGES = 3;

template <int MT, int NW, bool EDGE, int KC = 16>
__global__ void __launch_bounds__(NW * 32) k_gemm(GemmArgs g) {
    constexpr int NT = NW * 32, GBN = NW * 8, LDB_S = GBN + 4;  // GBN + 4 = 4 or 12 mod 16: conflict-free
    // k chunks of KC columns: 16 in a 3-stage ring, or 32 in a double buffer (half the barriers;
    // the launcher takes it where the chunks end exactly at Kp or at the rank-1 column)
    constexpr int HK = KC, HST = (KC == 32 ? 2 : GSTAGES), HLDA = (KC == 32 ? 36 : LDA_S);
    constexpr int NTL = MT + (EDGE ? 1 : 0);                     // accumulator tiles (+ the edge row)
    constexpr int AR = MT * 16 + (EDGE ? 1 : 0), ER = NTL * 16;  // A rows staged, epilogue row stride
    extern __shared__ double gsm[];
    double (*As)[AR][HLDA] = reinterpret_cast<double (*)[AR][HLDA]>(gsm);
    double (*Bs)[HK][LDB_S] = reinterpret_cast<double (*)[HK][LDB_S]>(gsm + HST * AR * HLDA);
    double* lrow = gsm + HST * (AR * HLDA + HK * LDB_S);  // [4][Kp]: d2hb, hb, d2ht, ht
    double* erow = lrow + 4 * g.Kp;  // [2][ER]: the epilogue's row factors (lam, or hb and ht)
    double* kcol = erow + 2 * ER;    // [AR][2]: A[r][K-1], A[r][K] of the rank-1 update
    double* krow = kcol + 2 * AR;    // [GBN]: B[K-1][c0 ..] of the rank-1 update
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gq = lane >> 2, tq = lane & 3;
    const int f = blockIdx.y;
    const long long c0 = (long long)blockIdx.x * GBN;
    const double* in = (f < 4 && g.inf[f]) ? g.inf[f] : g.in + f * g.in_fstride;
    const double* bcb = g.bcb ? g.bcb + f * g.bc_fstride : nullptr;
    const double* bct = g.bct ? g.bct + f * g.bc_fstride : nullptr;
    const bool lift = (g.epi != 5) && (bcb != nullptr);
    const int nchunks = (g.Kp + HK - 1) / HK;
    const bool edge_k = EDGE && !lift && nchunks > 1 && g.K == (nchunks - 1) * HK + 1;
    const int nmma = edge_k ? nchunks - 1 : nchunks;
    // tile MT of the EDGE form (the launcher guarantees M == 16 MT + 1): the edge row, row
    // MT*16 in its first two entries
    double acc[NTL][4];
#pragma unroll
    for (int t = 0; t < NTL; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
    double pe = 0.0;  // the edge row: this lane's partial sum for column warp*8 + gq

    // lifting: per-column factors of this lane's B column, per-row factors in shared memory
    // (zero past K, so the padded rows stay zero)
    const long long lc = c0 + warp * 8 + gq;
    double lbcb = 0.0, lbct = 0.0, lfac = 0.0;
    if (lift) {
        for (int k = tid; k < g.Kp; k += NT) {
            const bool ok = k < g.K;
            const int kin = k + g.koff;
            lrow[k] = ok ? g.d2hb[kin] : 0.0;
            lrow[g.Kp + k] = ok ? g.hb[kin] : 0.0;
            lrow[2 * g.Kp + k] = ok ? g.d2ht[kin] : 0.0;
            lrow[3 * g.Kp + k] = ok ? g.ht[kin] : 0.0;
        }
        if (lc < g.C) {
            lbcb = bcb[lc];
            lbct = bct[lc];
            lfac = (-w2_of(g, lc)) - g.lift_sigma;
        }
    }
    // the epilogue's row factors, staged once (their global loads would otherwise sit between
    // the stores of every output element)
    if (g.epi == EPI_HELM_SCALE || g.epi == EPI_LIFT_ADD) {
        for (int r = tid; r < ER; r += NT) {
            const bool ok = r < g.M;
            if (g.epi == EPI_HELM_SCALE) {
                erow[r] = ok ? g.lam[r] : 0.0;
            } else {
                erow[r] = ok ? g.hb[r + g.roff] : 0.0;
                erow[ER + r] = ok ? g.ht[r + g.roff] : 0.0;
            }
        }
    }
    constexpr int arows = AR;
    auto load_chunk = [&](int buf, int kc) {
        // A: 16-byte copies (Kp and the chunk start are multiples of 16 doubles)
        for (int idx = tid; idx < arows * (HK / 2); idx += NT) {
            const int r = idx / (HK / 2), cp = idx % (HK / 2);
            cp_async16(&As[buf][r][2 * cp], &g.A[(long long)r * g.Kp + kc + 2 * cp], 16);
        }
        // B: 16-byte copies of column pairs (C and the field stride are even)
        for (int idx = tid; idx < HK * (GBN / 2); idx += NT) {
            const int kk = idx / (GBN / 2), n2 = idx % (GBN / 2);
            const int k = kc + kk;
            const long long c = c0 + 2 * n2;
            const bool ok = (k < g.K && c < g.C);
            cp_async16(&Bs[buf][kk][2 * n2], ok ? (const void*)&in[(long long)(k + g.koff) * g.C + c] : (const void*)in,
                       ok ? 16 : 0);
        }
    };
    // B value of row k (chunk-relative kk) for this lane's column: raw, or lifted
    auto bval = [&](int buf, int kk, int k) {
        double v = Bs[buf][kk][warp * 8 + gq];
        if (lift) {
            const double abot = lrow[k] + lfac * lrow[g.Kp + k];
            v = v - abot * lbcb;
            const double atop = lrow[2 * g.Kp + k] + lfac * lrow[3 * g.Kp + k];
            v = v - atop * lbct;
        }
        return v;
    };

    // the rank-1 update's operands ride with the first chunk (16-byte pairs: K - 1, Kp and C
    // are even)
    const int kl = g.K - 1;
    if (EDGE && edge_k) {
        for (int r = tid; r < arows; r += NT) cp_async16(&kcol[2 * r], &g.A[(long long)r * g.Kp + kl], 16);
        for (int n2 = tid; n2 < GBN / 2; n2 += NT) {
            const long long c = c0 + 2 * n2;
            const bool ok = c < g.C;
            cp_async16(&krow[2 * n2], ok ? (const void*)&in[(long long)(kl + g.koff) * g.C + c] : (const void*)in,
                       ok ? 16 : 0);
        }
    }
#pragma unroll
    for (int st = 0; st < HST - 1; ++st) {
        if (st < nmma) load_chunk(st, st * HK);
        cp_async_commit();
    }
    for (int ch = 0; ch < nmma; ++ch) {
        const int buf = ch % HST;
        cp_async_wait<HST - 2>();
        __syncthreads();
        // the ring slot refilled here was read in iteration ch - 1, before the barrier
        if (ch + HST - 1 < nmma) load_chunk((ch + HST - 1) % HST, (ch + HST - 1) * HK);
        cp_async_commit();
#pragma unroll
        for (int k8 = 0; k8 < HK / 8; ++k8) {
            const int kk = k8 * 8 + tq;
            const double b0 = bval(buf, kk, ch * HK + kk);
            const double b1 = bval(buf, kk + 4, ch * HK + kk + 4);
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                const double a0 = As[buf][t * 16 + gq][k8 * 8 + tq];
                const double a1 = As[buf][t * 16 + gq + 8][k8 * 8 + tq];
                const double a2 = As[buf][t * 16 + gq][k8 * 8 + tq + 4];
                const double a3 = As[buf][t * 16 + gq + 8][k8 * 8 + tq + 4];
                dmma16(acc[t], a0, a1, a2, a3, b0, b1);
            }
            if constexpr (EDGE) {
                pe = fma(As[buf][AR - 1][kk], b0, pe);
                pe = fma(As[buf][AR - 1][kk + 4], b1, pe);
            }
        }
    }
    cp_async_wait<0>();
    const long long cb = c0 + warp * 8 + tq * 2;
    if (EDGE && edge_k) {
        // the last column of A against the last row of B (the lanes' own columns; zero-filled
        // past C)
        const double bq0 = krow[warp * 8 + 2 * tq], bq1 = krow[warp * 8 + 2 * tq + 1];
#pragma unroll
        for (int t = 0; t < MT; ++t) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const double a = kcol[2 * (t * 16 + hh * 8 + gq)];
                acc[t][2 * hh] = fma(a, bq0, acc[t][2 * hh]);
                acc[t][2 * hh + 1] = fma(a, bq1, acc[t][2 * hh + 1]);
            }
        }
        if (tq == 0) pe = fma(kcol[2 * (AR - 1)], krow[warp * 8 + gq], pe);
    }
    if constexpr (EDGE) {
        pe += __shfl_xor_sync(0xffffffffu, pe, 1);
        pe += __shfl_xor_sync(0xffffffffu, pe, 2);
        acc[NTL - 1][0] = __shfl_sync(0xffffffffu, pe, (2 * tq) * 4);
        acc[NTL - 1][1] = __shfl_sync(0xffffffffu, pe, (2 * tq + 1) * 4);
    }

    gemm_epilogue<NTL>(g, f, acc, 0, cb, gq, bcb, bct, erow, ER, g.M);
}

template <int MT, int NW, bool EDGE, int KC = 16>
size_t gemm_smem(int Kp) {
    constexpr int AR = MT * 16 + (EDGE ? 1 : 0), ER = (MT + (EDGE ? 1 : 0)) * 16;
    constexpr int HST = (KC == 32 ? 2 : GSTAGES), HLDA = (KC == 32 ? 36 : LDA_S);
    return (size_t)(HST * (AR * HLDA + KC * (NW * 8 + 4)) + 4 * Kp + 2 * ER + (EDGE ? 2 * AR + NW * 8 : 0)) *
           sizeof(double);
}

template <int MT, int NW, bool EDGE, int KC = 16>
void gemm_launch_t(const GemmArgs& g, cudaStream_t s) {
    const size_t sm = gemm_smem<MT, NW, EDGE, KC>(g.Kp);
    allow_smem((const void*)k_gemm<MT, NW, EDGE, KC>, sm);
    dim3 grid((unsigned)((g.C + NW * 8 - 1) / (NW * 8)), g.nfields);
    lsb::note_launch();
    k_gemm<MT, NW, EDGE, KC><<<grid, NW * 32, sm, s>>>(g);
}

// fraction of the last wave's slots that are busy, averaged over the waves
template <int MT, int NW, bool EDGE, int KC = 16>
double gemm_wave_eff(const GemmArgs& g) {
    const long long tiles = (g.C + NW * 8 - 1) / (NW * 8) * g.nfields;
    const long long slots =
        (long long)resident_blocks((const void*)k_gemm<MT, NW, EDGE, KC>, NW * 32, gemm_smem<MT, NW, EDGE, KC>(g.Kp)) *
        sm_count();
    if (slots <= 0) return 0.0;
    const long long waves = (tiles + slots - 1) / slots;
    return (double)tiles / (double)(waves * slots);
}

// 4..8 warps (32..64 columns) per CTA, whichever leaves the least idle in the last wave
// (ties to the wider CTA, which re-reads the matrix less)
template <int MT, bool EDGE, int KC = 16>
void gemm_pick(const GemmArgs& g, cudaStream_t s) {
    const double e8 = gemm_wave_eff<MT, 8, EDGE, KC>(g), e7 = gemm_wave_eff<MT, 7, EDGE, KC>(g),
                 e6 = gemm_wave_eff<MT, 6, EDGE, KC>(g), e5 = gemm_wave_eff<MT, 5, EDGE, KC>(g),
                 e4 = gemm_wave_eff<MT, 4, EDGE, KC>(g);
    double best = e8;
    int nw = 8;
    if (e7 > best + 0.02) best = e7, nw = 7;
    if (e6 > best + 0.02) best = e6, nw = 6;
    if (e5 > best + 0.02) best = e5, nw = 5;
    if (e4 > best + 0.02) best = e4, nw = 4;
    if (g.nw >= 4 && g.nw <= 8) nw = g.nw;  // a tuned schedule overrides the model
    switch (nw) {
        case 8: gemm_launch_t<MT, 8, EDGE, KC>(g, s); break;
        case 7: gemm_launch_t<MT, 7, EDGE, KC>(g, s); break;
        case 6: gemm_launch_t<MT, 6, EDGE, KC>(g, s); break;
        case 5: gemm_launch_t<MT, 5, EDGE, KC>(g, s); break;
        default: gemm_launch_t<MT, 4, EDGE, KC>(g, s); break;
    }
}

// Small grids: k_gemm gives every warp all row tiles of its columns and has one chunk of loads
// in flight, so that a few thousand columns leave most SMs idle while a few walk the whole
// matrix.  Here a CTA of 4 warps takes GS_RT row tiles of 32 columns, with the whole k range
// of both operands in shared memory, requested up front in two halves.  The sums are k_gemm's,
// in its order: the tiles in k steps of 8, the EDGE forms' last column as the rank-1 update and
// their last row on the FP64 pipe (by the CTAs of the last row tiles).  Bound by latency (launch,
// one round of loads, a chain of K/8 MMAs); measured per launch, the step's four: 512 columns,
// nz 96: 13.2-17.1 -> 7.0 us; 1024 columns, nz 64: 8.3 -> 6.5 us on average.
constexpr int GS_RT = 2, GS_NW = 4;

template <bool EDGE>
__global__ void __launch_bounds__(GS_NW * 32) k_gemm_s(GemmArgs g, int mt) {
    constexpr int NT = GS_NW * 32, GBN = GS_NW * 8, LDB = GBN + 4, NTL = GS_RT + (EDGE ? 1 : 0), AR = GS_RT * 16 + 1;
    extern __shared__ double gsm[];
    const int lda = g.Kp + 4;                   // 4 mod 16: conflict-free
    double* As = gsm;                           // [AR][lda]: the CTA's rows, then the edge row
    double* Bs = As + AR * lda;                 // [Kp][LDB]
    double* lrow = Bs + (size_t)g.Kp * LDB;     // [4][Kp]: d2hb, hb, d2ht, ht
    double* erow = lrow + 4 * g.Kp;             // [2][ER]
    constexpr int ER = NTL * 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gq = lane >> 2, tq = lane & 3;
    const int f = blockIdx.y;
    const int t0 = blockIdx.z * GS_RT, nt = min(GS_RT, mt - t0);
    const bool edge = EDGE && t0 + nt == mt;    // this CTA carries the edge row
    const long long c0 = (long long)blockIdx.x * GBN;
    const double* in = (f < 4 && g.inf[f]) ? g.inf[f] : g.in + f * g.in_fstride;
    const double* bcb = g.bcb ? g.bcb + f * g.bc_fstride : nullptr;
    const double* bct = g.bct ? g.bct + f * g.bc_fstride : nullptr;
    const bool lift = (g.epi != EPI_LIFT_ADD) && (bcb != nullptr);
    const bool edge_k = EDGE && !lift && g.K > 16 && g.K % 16 == 1;
    const int km = edge_k ? g.K - 1 : g.Kp;     // k range of the MMAs, a multiple of 16
    const int half = (km / 2 + 7) & ~7;

    auto load = [&](int ka, int kb) {           // operands of k rows [ka, kb), multiples of 2
        const int np = (kb - ka) / 2;
        const int nr = nt * 16 + (edge ? 1 : 0);
        for (int idx = tid; idx < nr * np; idx += NT) {
            const int r = idx / np, k = ka + 2 * (idx - r * np);
            const int lr = r < nt * 16 ? r : AR - 1;
            const long long gr = r < nt * 16 ? t0 * 16 + r : mt * 16;
            cp_async16(&As[lr * lda + k], &g.A[gr * g.Kp + k], 16);
        }
        for (int idx = tid; idx < (kb - ka) * (GBN / 2); idx += NT) {
            const int k = ka + idx / (GBN / 2), n2 = idx % (GBN / 2);
            const long long c = c0 + 2 * n2;
            const bool ok = (k < g.K && c < g.C);
            cp_async16(&Bs[k * LDB + 2 * n2], ok ? (const void*)&in[(long long)(k + g.koff) * g.C + c] : (const void*)in,
                       ok ? 16 : 0);
        }
    };
    load(0, half);
    cp_async_commit();
    load(half, edge_k ? km + 2 : km);           // the rank-1 column and row ride along (K + 1 <= Kp)
    cp_async_commit();

    const long long lc = c0 + warp * 8 + gq;
    const long long cb = c0 + warp * 8 + tq * 2;
    double lbcb = 0.0, lbct = 0.0, lfac = 0.0;
    if (lift) {
        for (int k = tid; k < g.Kp; k += NT) {
            const bool ok = k < g.K;
            const int kin = k + g.koff;
            lrow[k] = ok ? g.d2hb[kin] : 0.0;
            lrow[g.Kp + k] = ok ? g.hb[kin] : 0.0;
            lrow[2 * g.Kp + k] = ok ? g.d2ht[kin] : 0.0;
            lrow[3 * g.Kp + k] = ok ? g.ht[kin] : 0.0;
        }
        if (lc < g.C) {
            lbcb = bcb[lc];
            lbct = bct[lc];
            lfac = (-w2_of(g, lc)) - g.lift_sigma;
        }
    }
    if (g.epi == EPI_HELM_SCALE || g.epi == EPI_LIFT_ADD) {
        for (int i = tid; i < ER; i += NT) {
            const int r = t0 * 16 + i;
            const bool ok = r < g.M;
            if (g.epi == EPI_HELM_SCALE) {
                erow[i] = ok ? g.lam[r] : 0.0;
            } else {
                erow[i] = ok ? g.hb[r + g.roff] : 0.0;
                erow[ER + i] = ok ? g.ht[r + g.roff] : 0.0;
            }
        }
    }

    double acc[NTL][4];
#pragma unroll
    for (int t = 0; t < NTL; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
    double pe = 0.0;
    auto steps = [&](int ka, int kb) {
#pragma unroll 4
        for (int k = ka; k < kb; k += 8) {
            double b[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int kk = k + 4 * h + tq;
                double v = Bs[kk * LDB + warp * 8 + gq];
                if (lift) {
                    const double abot = lrow[kk] + lfac * lrow[g.Kp + kk];
                    v = v - abot * lbcb;
                    const double atop = lrow[2 * g.Kp + kk] + lfac * lrow[3 * g.Kp + kk];
                    v = v - atop * lbct;
                }
                b[h] = v;
            }
#pragma unroll
            for (int t = 0; t < GS_RT; ++t) {
                if (t >= nt) break;
                const double* a = &As[(t * 16 + gq) * lda + k + tq];
                dmma16(acc[t], a[0], a[8 * lda], a[4], a[8 * lda + 4], b[0], b[1]);
            }
            if (EDGE && edge) {
                pe = fma(As[(AR - 1) * lda + k + tq], b[0], pe);
                pe = fma(As[(AR - 1) * lda + k + tq + 4], b[1], pe);
            }
        }
    };
    cp_async_wait<1>();
    __syncthreads();
    steps(0, half);
    cp_async_wait<0>();
    __syncthreads();
    steps(half, km);
    if (EDGE && edge_k) {
        const double* kr = &Bs[km * LDB + warp * 8];
        const double bq0 = kr[2 * tq], bq1 = kr[2 * tq + 1];
#pragma unroll
        for (int t = 0; t < GS_RT; ++t) {
            if (t >= nt) break;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const double a = As[(t * 16 + hh * 8 + gq) * lda + km];
                acc[t][2 * hh] = fma(a, bq0, acc[t][2 * hh]);
                acc[t][2 * hh + 1] = fma(a, bq1, acc[t][2 * hh + 1]);
            }
        }
        if (edge && tq == 0) pe = fma(As[(AR - 1) * lda + km], kr[gq], pe);
    }
    if constexpr (EDGE) {
        if (edge) {  // the edge row is the tile after this CTA's last
            pe += __shfl_xor_sync(0xffffffffu, pe, 1);
            pe += __shfl_xor_sync(0xffffffffu, pe, 2);
            const double e0 = __shfl_sync(0xffffffffu, pe, (2 * tq) * 4);
            const double e1 = __shfl_sync(0xffffffffu, pe, (2 * tq + 1) * 4);
#pragma unroll
            for (int t = 1; t < NTL; ++t)
                if (t == nt) {
                    acc[t][0] = e0;
                    acc[t][1] = e1;
                }
        }
    }
    gemm_epilogue<NTL>(g, f, acc, t0, cb, gq, bcb, bct, erow, ER, edge ? g.M : min(g.M, (t0 + nt) * 16));
}

// 32-column tiles of a contraction over all its fields: at most one per SM takes the kernels
// for small grids.  Beyond that the large-grid kernels' better reuse wins (three fields of 4096
// columns, nz 64: solve 16.4 us large, 14.8 small, but the contractions 9.0 and 11.9 against
// 10.3 each, and a run beside others 217 -> 221 us a step)
bool small_grid(const GemmArgs& g) { return g.nw == 0 && (g.C + 31) / 32 * g.nfields <= sm_count(); }

template <bool EDGE>
void gemm_small_t(const GemmArgs& g, int mt, cudaStream_t s) {
    const size_t sm = ((size_t)(GS_RT * 16 + 1) * (g.Kp + 4) + (size_t)g.Kp * (GS_NW * 8 + 4) + 4 * g.Kp +
                       2 * (GS_RT + 1) * 16) * sizeof(double);
    allow_smem((const void*)k_gemm_s<EDGE>, sm);
    dim3 grid((unsigned)((g.C + GS_NW * 8 - 1) / (GS_NW * 8)), g.nfields, (mt + GS_RT - 1) / GS_RT);
    lsb::note_launch();
    k_gemm_s<EDGE><<<grid, GS_NW * 32, sm, s>>>(g, mt);
}

void launch_gemm(const GemmArgs& g, cudaStream_t s) {
    // M = 16 MT + 1 (nzp = 2^n + 1): MT tiles and the edge row, not a mostly-zero last tile
    // (at 256x64x129: dz of u, v, w 90.6 -> 78.4 us, dz of h_l3 with the divergence 111 ->
    // 102.8 us)
    const int mt = g.Mp / 16 - 1;
    const bool edge = g.M == mt * 16 + 1 && (mt == 1 || mt == 2 || mt == 4 || mt == 8);
    // (with more than two CTAs of k_gemm_s per SM the right-hand sides, read by every row group,
    // cost what the even spread gives: 4096 columns, nz 96: 19.2 -> 12.5 us alone, but 380 ->
    // 394 us a step beside other runs)
    if (small_grid(g) && (g.C + 31) / 32 * g.nfields * ((mt + (edge ? 0 : 1) + GS_RT - 1) / GS_RT) <= 2LL * sm_count()) {
        edge ? gemm_small_t<true>(g, mt, s) : gemm_small_t<false>(g, mt + 1, s);
        return;
    }
    if (edge) {
        // k chunks of 32 where they end exactly at Kp, or at the rank-1 column, for the light
        // epilogues (at 256x64x129: dz of u, v, w 80.3 -> 77.4 us, the Poisson right-hand side
        // -1.8 us; the divergence and pressure epilogues, which read three fields per element,
        // measured slower with them, 103 -> 121 and 47 -> 52 us)
        const bool lift = g.epi != EPI_LIFT_ADD && g.bcb != nullptr;
        const bool k32 = (g.epi == EPI_STORE || g.epi == EPI_POISSON_RHS) &&
                         (g.Kp % 32 == 0 || (!lift && g.K == g.Kp - 15 && (g.Kp - 16) % 32 == 0));
        switch (mt) {
            case 1: gemm_pick<1, true>(g, s); return;
            case 2: gemm_pick<2, true>(g, s); return;
            case 4: k32 ? gemm_pick<4, true, 32>(g, s) : gemm_pick<4, true>(g, s); return;
            case 8: k32 ? gemm_pick<8, true, 32>(g, s) : gemm_pick<8, true>(g, s); return;
            default: break;
        }
    }
    switch (g.Mp / 16) {
#define LSB_MT(n) \
    case n: gemm_pick<n, false>(g, s); break;
        LSB_MT(1) LSB_MT(2) LSB_MT(3) LSB_MT(4) LSB_MT(5) LSB_MT(6) LSB_MT(7) LSB_MT(8) LSB_MT(9)
#undef LSB_MT
        default: break;
    }
}

// The Helmholtz solve in one launch (src/helmholtz.f90:130-208 with the lifting of :324-353):
// Y = E^-1 (rhs - lift) scaled by 1/(lam_r - k^2 - sigma), then out = E Y + hb bcb + ht bct on
// the interior rows and the lift alone on the ceiling and wall rows (E has no rows there).
// Both matrices are zero-padded to KP = 16 MT1 >= nzm rows and columns, so every nz has this
// form; the intermediate never goes to memory.  Every product and sum is the one two separate
// contractions make, in the same order, whichever kernel below runs.

// 16 bytes by cp.async (zeros where !ok), in two 8-byte copies when the source field of a
// caller's own memory is not 16-byte aligned
__device__ __forceinline__ void cp_async_pair(double* d, const double* src, const double* safe, bool ok, bool al16) {
    if (al16) {
        cp_async16(d, ok ? src : safe, ok ? 16 : 0);
    } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const unsigned sa = (unsigned)__cvta_generic_to_shared(d + e);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(ok ? src + e : safe), "r"(ok ? 8 : 0));
        }
    }
}
__device__ __forceinline__ void store_pair(double* o, double v0, double v1, bool al16) {
    if (al16) {
        *reinterpret_cast<double2*>(o) = make_double2(v0, v1);
    } else {
        o[0] = v0;
        o[1] = v1;
    }
}
__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<unsigned long long>(p) & 15) == 0; }

// the ceiling (row 0) and wall rows of the solution: the lift alone
__device__ __forceinline__ void helm_boundary_row(const GemmArgs& g2, double* out, bool wall, long long cb,
                                                  const double (&eb)[2], const double (&et)[2], bool lift, bool al16) {
    const int row = wall ? g2.M + 1 : 0;
    double v0 = 0.0, v1 = 0.0;
    if (lift) {
        const double hb = g2.hb[row], ht = g2.ht[row];
        v0 = v0 + hb * eb[0] + ht * et[0];
        v1 = v1 + hb * eb[1] + ht * et[1];
    }
    store_pair(out + (long long)row * g2.C + cb, v0, v1, al16);
}

// Large grids.  The CTA's Y block (all KP rows x its 8 NW columns) stays in the accumulator
// registers of the first contraction and feeds the second as its B operand through warp
// shuffles.  The second contraction runs in two row passes (registers: Y plus half of the
// output tiles); its A chunks continue the first contraction's cp.async ring.
//
// B regrouping: the second contraction's fragment b0 = Y[k = 16 ch + 8 k8 + tq][n = gq] of
// lane (gq, tq) sits in accumulator acc[ch][2 k8 + (gq & 1)] of lane 4 tq + gq / 2 (the
// accumulator holds D[8 (q / 2) + gq'][2 tq' + (q & 1)]); b1 is the row 4 further on, in lane
// 4 (tq + 4) + gq / 2.
template <int MT1, int NW, int KC>
__global__ void __launch_bounds__(NW * 32, 2) k_helm(GemmArgs g1, GemmArgs g2) {
    constexpr int NT = NW * 32, GBN = NW * 8, LDB_S = GBN + 4;
    constexpr int P2A = (MT1 + 1) / 2, P2B = MT1 - P2A;  // output row tiles of the two passes
    // k chunks of KC columns: 16 in a 3-stage ring, or 32 in a double buffer (half the
    // barriers per contraction)
    constexpr int HK = KC, HST = (KC == 32 ? 2 : GSTAGES), HLDA = (KC == 32 ? 36 : LDA_S);
    constexpr int NCH = MT1 * 16 / KC;                   // k chunks per contraction (Kp = 16 MT1)
    constexpr int NTOT = NCH * (P2B > 0 ? 3 : 2);
    constexpr int KP = MT1 * 16;
    extern __shared__ double gsm[];
    double (*As)[KP][HLDA] = reinterpret_cast<double (*)[KP][HLDA]>(gsm);
    double (*Bs)[HK][LDB_S] = reinterpret_cast<double (*)[HK][LDB_S]>(gsm + HST * KP * HLDA);
    double* lrow = gsm + HST * (KP * HLDA + HK * LDB_S);  // [4][KP]: d2hb, hb, d2ht, ht
    double* elam = lrow + 4 * KP;                         // [KP]
    double* ehb = elam + KP;                              // [KP]
    double* eht = ehb + KP;                               // [KP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gq = lane >> 2, tq = lane & 3;
    const int f = blockIdx.y;
    const long long C = g1.C;
    const long long c0 = (long long)blockIdx.x * GBN;
    const double* in = (f < 4 && g1.inf[f]) ? g1.inf[f] : g1.in + f * g1.in_fstride;
    const double* bcb = g1.bcb ? g1.bcb + f * g1.bc_fstride : nullptr;
    const double* bct = g1.bct ? g1.bct + f * g1.bc_fstride : nullptr;
    const bool lift = bcb != nullptr;
    const bool in16 = aligned16(in);

    const long long lc = c0 + warp * 8 + gq;
    double lbcb = 0.0, lbct = 0.0, lfac = 0.0;
    if (lift) {
        for (int k = tid; k < KP; k += NT) {
            const bool ok = k < g1.K;
            const int kin = k + g1.koff;
            lrow[k] = ok ? g1.d2hb[kin] : 0.0;
            lrow[KP + k] = ok ? g1.hb[kin] : 0.0;
            lrow[2 * KP + k] = ok ? g1.d2ht[kin] : 0.0;
            lrow[3 * KP + k] = ok ? g1.ht[kin] : 0.0;
            ehb[k] = (k < g2.M) ? g2.hb[k + g2.roff] : 0.0;
            eht[k] = (k < g2.M) ? g2.ht[k + g2.roff] : 0.0;
        }
        if (lc < C) {
            lbcb = bcb[lc];
            lbct = bct[lc];
            lfac = (-w2_of(g1, lc)) - g1.lift_sigma;
        }
    }
    for (int r = tid; r < KP; r += NT) elam[r] = r < g1.M ? g1.lam[r] : 0.0;

    // chunk gc of the ring: E^-1 with the right-hand side for gc < NCH, then E's rows of
    // pass 0 and of pass 1
    auto issue = [&](int gc) {
        const int buf = gc % HST;
        if (gc < NCH) {
            const int kc = gc * HK;
            for (int idx = tid; idx < MT1 * 16 * (HK / 2); idx += NT) {
                const int r = idx / (HK / 2), cp = idx % (HK / 2);
                cp_async16(&As[buf][r][2 * cp], &g1.A[(long long)r * KP + kc + 2 * cp], 16);
            }
            for (int idx = tid; idx < HK * (GBN / 2); idx += NT) {
                const int kk = idx / (GBN / 2), n2 = idx % (GBN / 2);
                const int k = kc + kk;
                const long long c = c0 + 2 * n2;
                cp_async_pair(&Bs[buf][kk][2 * n2], &in[(long long)(k + g1.koff) * C + c], in, k < g1.K && c < C, in16);
            }
        } else {
            const int p = (gc - NCH) / NCH;
            const int kc = ((gc - NCH) % NCH) * HK;
            const int r0 = p ? P2A * 16 : 0;
            const int nr = p ? P2B * 16 : P2A * 16;
            for (int idx = tid; idx < nr * (HK / 2); idx += NT) {
                const int r = idx / (HK / 2), cp = idx % (HK / 2);
                cp_async16(&As[buf][r][2 * cp], &g2.A[(long long)(r0 + r) * KP + kc + 2 * cp], 16);
            }
        }
    };
    // the slot refilled here was read in iteration gc - 1, before the barrier
    auto advance = [&](int gc) {
        cp_async_wait<HST - 2>();
        __syncthreads();
        if (gc + HST - 1 < NTOT) issue(gc + HST - 1);
        cp_async_commit();
    };
    auto bval = [&](int buf, int kk, int k) {
        double v = Bs[buf][kk][warp * 8 + gq];
        if (lift) {
            const double abot = lrow[k] + lfac * lrow[KP + k];
            v = v - abot * lbcb;
            const double atop = lrow[2 * KP + k] + lfac * lrow[3 * KP + k];
            v = v - atop * lbct;
        }
        return v;
    };

    double acc[MT1][4];
#pragma unroll
    for (int t = 0; t < MT1; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
#pragma unroll
    for (int st = 0; st < HST - 1; ++st) {
        if (st < NTOT) issue(st);
        cp_async_commit();
    }
    for (int ch = 0; ch < NCH; ++ch) {
        advance(ch);
        const int buf = ch % HST;
#pragma unroll
        for (int k8 = 0; k8 < HK / 8; ++k8) {
            const int kk = k8 * 8 + tq;
            const double b0 = bval(buf, kk, ch * HK + kk);
            const double b1 = bval(buf, kk + 4, ch * HK + kk + 4);
#pragma unroll
            for (int t = 0; t < MT1; ++t) {
                const double a0 = As[buf][t * 16 + gq][k8 * 8 + tq];
                const double a1 = As[buf][t * 16 + gq + 8][k8 * 8 + tq];
                const double a2 = As[buf][t * 16 + gq][k8 * 8 + tq + 4];
                const double a3 = As[buf][t * 16 + gq + 8][k8 * 8 + tq + 4];
                dmma16(acc[t], a0, a1, a2, a3, b0, b1);
            }
        }
    }

    // Y = acc / (lam_r - k^2 - sigma); the padded rows and columns are zero
    const long long cb = c0 + warp * 8 + tq * 2;
    double ew2[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e)
        if (cb + e < C) ew2[e] = w2_of(g1, cb + e);
#pragma unroll
    for (int t = 0; t < MT1; ++t) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = t * 16 + (q >> 1) * 8 + gq;
            const int e = q & 1;
            const double dfac = (-ew2[e]) - g1.sigma;
            acc[t][q] = (r < g1.M && cb + e < C) ? acc[t][q] / (elam[r] + dfac) : 0.0;
        }
    }

    double* __restrict__ out = (f < 4 && g2.outf[f]) ? g2.outf[f] : g2.out + f * g2.out_fstride;
    const bool out16 = aligned16(out);
    double eb[2] = {0.0, 0.0}, et[2] = {0.0, 0.0};
    if (lift && cb < C) {
        eb[0] = bcb[cb];
        eb[1] = bcb[cb + 1];
        et[0] = bct[cb];
        et[1] = bct[cb + 1];
    }
    if (cb < C && gq < 2) helm_boundary_row(g2, out, gq == 1, cb, eb, et, lift, out16);
    const int src0 = tq * 4 + (gq >> 1), src1 = (tq + 4) * 4 + (gq >> 1);
    const bool odd = (gq & 1) != 0;
    // one pass over output row tiles TB .. TB + P - 1 of E Y, then its store
    auto pass = [&](auto tb_c, auto p_c) {
        constexpr int TB = decltype(tb_c)::value, P = decltype(p_c)::value;
        double acc2[P][4];
#pragma unroll
        for (int t = 0; t < P; ++t) acc2[t][0] = acc2[t][1] = acc2[t][2] = acc2[t][3] = 0.0;
        constexpr int G0 = NCH * (TB == 0 ? 1 : 2);
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
            advance(G0 + ch);
            const int buf = (G0 + ch) % HST;
#pragma unroll
            for (int k8 = 0; k8 < HK / 8; ++k8) {
                // rows 8 k8 .. of chunk ch are rows 8 (k8 % 2) .. of Y tile ch * KC / 16 + k8 / 2
                const int yt = ch * (HK / 16) + (k8 >> 1), yk = k8 & 1;
                const double l0 = __shfl_sync(0xffffffffu, acc[yt][2 * yk], src0);
                const double h0 = __shfl_sync(0xffffffffu, acc[yt][2 * yk + 1], src0);
                const double l1 = __shfl_sync(0xffffffffu, acc[yt][2 * yk], src1);
                const double h1 = __shfl_sync(0xffffffffu, acc[yt][2 * yk + 1], src1);
                const double b0 = odd ? h0 : l0, b1 = odd ? h1 : l1;
#pragma unroll
                for (int t = 0; t < P; ++t) {
                    const double a0 = As[buf][t * 16 + gq][k8 * 8 + tq];
                    const double a1 = As[buf][t * 16 + gq + 8][k8 * 8 + tq];
                    const double a2 = As[buf][t * 16 + gq][k8 * 8 + tq + 4];
                    const double a3 = As[buf][t * 16 + gq + 8][k8 * 8 + tq + 4];
                    dmma16(acc2[t], a0, a1, a2, a3, b0, b1);
                }
            }
        }
        if (cb >= C) return;  // C and cb are even: cb < C covers both columns
#pragma unroll
        for (int t = 0; t < P; ++t) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int r = (TB + t) * 16 + hh * 8 + gq;
                if (r >= g2.M) continue;
                double v0 = acc2[t][2 * hh], v1 = acc2[t][2 * hh + 1];
                if (lift) {
                    v0 = v0 + ehb[r] * eb[0] + eht[r] * et[0];
                    v1 = v1 + ehb[r] * eb[1] + eht[r] * et[1];
                }
                store_pair(out + (long long)(r + g2.roff) * C + cb, v0, v1, out16);
            }
        }
    };
    pass(std::integral_constant<int, 0>{}, std::integral_constant<int, P2A>{});
    if constexpr (P2B > 0) pass(std::integral_constant<int, P2A>{}, std::integral_constant<int, P2B>{});
    cp_async_wait<0>();
}

// Small grids: too few columns to give every SM a CTA of k_helm, whose warps each walk all row
// tiles of both products behind one chunk of loads in flight.  Here a CTA owns 8 NC columns and
// NR warps share each of them, a warp taking every NR-th part of the row tiles; all chunks that
// fit shared memory are requested up front, and Y passes between the warps through the
// right-hand side's buffer.  Bound by latency; measured: three fields of 512 columns at nz 96
// 29.7 us (two contractions) -> 9.4, one field 33.2 -> 9.5; nz 64, three fields of 1024 columns
// 12.9 (k_helm) -> 8.4, one field 12.9 -> 5.8; one field of 4096 columns 14.6 -> 8.3.
constexpr size_t kHelmSmallSmem = 112 * 1024;  // two CTAs per SM

template <int MT1, int NC>
struct HelmSmall {
    static constexpr int NR0 = (NC == 4 ? 2 : 4), NR = MT1 < NR0 ? MT1 : NR0;
    static constexpr int TPW = (MT1 + NR - 1) / NR;          // row tiles per warp
    static constexpr int NT = NC * NR * 32;
    static constexpr int KP = MT1 * 16, KC = (MT1 % 2 == 0 && MT1 <= 6) ? 32 : 16;
    static constexpr int LDA = KC + 4, LDB = NC * 8 + 4;     // 4 or 12 mod 16: conflict-free
    static constexpr int NCH = KP / KC, NTOT = 2 * NCH;      // chunks of E^-1, then of E
    static constexpr size_t fixed = (size_t)(KP * LDB + 7 * KP) * sizeof(double);
    static constexpr size_t stage = (size_t)KP * LDA * sizeof(double);
    static constexpr int fit = (int)((kHelmSmallSmem - fixed) / stage);
    static constexpr int HST = fit < NTOT ? fit : NTOT;      // stages of the chunk ring
    static constexpr size_t smem = HST * stage + fixed;
    static_assert(HST >= 2, "chunk ring");
};

template <int MT1, int NC>
__global__ void __launch_bounds__(HelmSmall<MT1, NC>::NT) k_helm_s(GemmArgs g1, GemmArgs g2) {
    using L = HelmSmall<MT1, NC>;
    constexpr int KP = L::KP, KC = L::KC, NCH = L::NCH, HST = L::HST, TPW = L::TPW, NT = L::NT, GBN = NC * 8;
    extern __shared__ double gsm[];
    double (*As)[KP][L::LDA] = reinterpret_cast<double (*)[KP][L::LDA]>(gsm);
    double (*Bs)[L::LDB] = reinterpret_cast<double (*)[L::LDB]>(gsm + HST * KP * L::LDA);  // rhs, then Y
    double* lrow = &Bs[KP][0];       // [4][KP]: d2hb, hb, d2ht, ht
    double* elam = lrow + 4 * KP;    // [KP]
    double* ehb = elam + KP;         // [KP]
    double* eht = ehb + KP;          // [KP]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wc = warp % NC, wr = warp / NC;
    const int gq = lane >> 2, tq = lane & 3;
    const int f = blockIdx.y;
    const long long C = g1.C;
    const long long c0 = (long long)blockIdx.x * GBN;
    const double* in = (f < 4 && g1.inf[f]) ? g1.inf[f] : g1.in + f * g1.in_fstride;
    const double* bcb = g1.bcb ? g1.bcb + f * g1.bc_fstride : nullptr;
    const double* bct = g1.bct ? g1.bct + f * g1.bc_fstride : nullptr;
    const bool lift = bcb != nullptr;
    const bool in16 = aligned16(in);

    auto issue = [&](int gc) {
        const int buf = gc % HST;
        const bool first = gc < NCH;
        const double* A = first ? g1.A : g2.A;
        const int kc = (first ? gc : gc - NCH) * KC;
        for (int idx = tid; idx < KP * (KC / 2); idx += NT) {
            const int r = idx / (KC / 2), cp = idx % (KC / 2);
            cp_async16(&As[buf][r][2 * cp], &A[(long long)r * KP + kc + 2 * cp], 16);
        }
        if (first) {
            for (int idx = tid; idx < KC * (GBN / 2); idx += NT) {
                const int kk = idx / (GBN / 2), n2 = idx % (GBN / 2);
                const int k = kc + kk;
                const long long c = c0 + 2 * n2;
                cp_async_pair(&Bs[k][2 * n2], &in[(long long)(k + g1.koff) * C + c], in, k < g1.K && c < C, in16);
            }
        }
    };
#pragma unroll
    for (int st = 0; st < HST - 1; ++st) {
        issue(st);
        cp_async_commit();
    }
    // the slot refilled here was read in iteration gc - 1, before the barrier
    auto advance = [&](int gc) {
        cp_async_wait<HST - 2>();
        __syncthreads();
        if (gc + HST - 1 < L::NTOT) issue(gc + HST - 1);
        cp_async_commit();
    };

    const long long lc = c0 + wc * 8 + gq;
    const long long cb = c0 + wc * 8 + tq * 2;
    double lbcb = 0.0, lbct = 0.0, lfac = 0.0;
    double eb[2] = {0.0, 0.0}, et[2] = {0.0, 0.0};
    if (lift) {
        for (int k = tid; k < KP; k += NT) {
            const bool ok = k < g1.K;
            const int kin = k + g1.koff;
            lrow[k] = ok ? g1.d2hb[kin] : 0.0;
            lrow[KP + k] = ok ? g1.hb[kin] : 0.0;
            lrow[2 * KP + k] = ok ? g1.d2ht[kin] : 0.0;
            lrow[3 * KP + k] = ok ? g1.ht[kin] : 0.0;
            ehb[k] = (k < g2.M) ? g2.hb[k + g2.roff] : 0.0;
            eht[k] = (k < g2.M) ? g2.ht[k + g2.roff] : 0.0;
        }
        if (lc < C) {
            lbcb = bcb[lc];
            lbct = bct[lc];
            lfac = (-w2_of(g1, lc)) - g1.lift_sigma;
        }
        if (cb < C) {
            eb[0] = bcb[cb];
            eb[1] = bcb[cb + 1];
            et[0] = bct[cb];
            et[1] = bct[cb + 1];
        }
    }
    for (int r = tid; r < KP; r += NT) elam[r] = r < g1.M ? g1.lam[r] : 0.0;
    double ew2[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e)
        if (cb + e < C) ew2[e] = w2_of(g1, cb + e);

    // one product over this warp's row tiles wr TPW .. (those below MT1)
    double acc[TPW][4];
    auto product = [&](int g0, bool lifted) {
#pragma unroll
        for (int t = 0; t < TPW; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
        for (int ch = 0; ch < NCH; ++ch) {
            advance(g0 + ch);
            const int buf = (g0 + ch) % HST;
#pragma unroll
            for (int k8 = 0; k8 < KC / 8; ++k8) {
                double b[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int k = ch * KC + k8 * 8 + h * 4 + tq;
                    double v = Bs[k][wc * 8 + gq];
                    if (lifted) {
                        const double abot = lrow[k] + lfac * lrow[KP + k];
                        v = v - abot * lbcb;
                        const double atop = lrow[2 * KP + k] + lfac * lrow[3 * KP + k];
                        v = v - atop * lbct;
                    }
                    b[h] = v;
                }
#pragma unroll
                for (int t = 0; t < TPW; ++t) {
                    const int tt = wr * TPW + t;
                    if (MT1 % L::NR != 0 && tt >= MT1) break;
                    const double a0 = As[buf][tt * 16 + gq][k8 * 8 + tq];
                    const double a1 = As[buf][tt * 16 + gq + 8][k8 * 8 + tq];
                    const double a2 = As[buf][tt * 16 + gq][k8 * 8 + tq + 4];
                    const double a3 = As[buf][tt * 16 + gq + 8][k8 * 8 + tq + 4];
                    dmma16(acc[t], a0, a1, a2, a3, b[0], b[1]);
                }
            }
        }
    };
    product(0, lift);
    __syncthreads();  // every warp has read the right-hand side: its buffer becomes Y
#pragma unroll
    for (int t = 0; t < TPW; ++t) {
        const int tt = wr * TPW + t;
        if (tt >= MT1) break;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = tt * 16 + (q >> 1) * 8 + gq;
            const int e = q & 1;
            const double dfac = (-ew2[e]) - g1.sigma;
            Bs[r][wc * 8 + tq * 2 + e] = (r < g1.M && cb + e < C) ? acc[t][q] / (elam[r] + dfac) : 0.0;
        }
    }
    product(NCH, false);  // its first barrier orders Y
    cp_async_wait<0>();
    if (cb >= C) return;
    double* __restrict__ out = (f < 4 && g2.outf[f]) ? g2.outf[f] : g2.out + f * g2.out_fstride;
    const bool out16 = aligned16(out);
    if (wr == 0 && gq < 2) helm_boundary_row(g2, out, gq == 1, cb, eb, et, lift, out16);
#pragma unroll
    for (int t = 0; t < TPW; ++t) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int r = (wr * TPW + t) * 16 + hh * 8 + gq;
            if (r >= g2.M) continue;
            double v0 = acc[t][2 * hh], v1 = acc[t][2 * hh + 1];
            if (lift) {
                v0 = v0 + ehb[r] * eb[0] + eht[r] * et[0];
                v1 = v1 + ehb[r] * eb[1] + eht[r] * et[1];
            }
            store_pair(out + (long long)(r + g2.roff) * C + cb, v0, v1, out16);
        }
    }
}

template <int MT1, int NW, int KC>
size_t helm_smem() {
    constexpr int HST = (KC == 32 ? 2 : GSTAGES), HLDA = (KC == 32 ? 36 : LDA_S);
    return (size_t)(HST * (MT1 * 16 * HLDA + KC * (NW * 8 + 4)) + 7 * MT1 * 16) * sizeof(double);
}

template <int MT1, int NW, int KC>
double helm_wave_eff(const GemmArgs& g) {
    const long long tiles = (g.C + NW * 8 - 1) / (NW * 8) * g.nfields;
    const long long slots =
        (long long)resident_blocks((const void*)k_helm<MT1, NW, KC>, NW * 32, helm_smem<MT1, NW, KC>()) * sm_count();
    if (slots <= 0) return 0.0;
    const long long waves = (tiles + slots - 1) / slots;
    return (double)tiles / (double)(waves * slots);
}

template <int MT1, int NW, int KC>
bool helm_launch_t(const GemmArgs& g1, const GemmArgs& g2, cudaStream_t s) {
    const size_t sm = helm_smem<MT1, NW, KC>();
    if (!allow_smem((const void*)k_helm<MT1, NW, KC>, sm)) return false;
    dim3 grid((unsigned)((g1.C + NW * 8 - 1) / (NW * 8)), g1.nfields);
    lsb::note_launch();
    k_helm<MT1, NW, KC><<<grid, NW * 32, sm, s>>>(g1, g2);
    return true;
}

template <int MT1, int NC>
bool helm_small_t(const GemmArgs& g1, const GemmArgs& g2, cudaStream_t s) {
    using L = HelmSmall<MT1, NC>;
    if (!allow_smem((const void*)k_helm_s<MT1, NC>, L::smem)) return false;
    dim3 grid((unsigned)((g1.C + NC * 8 - 1) / (NC * 8)), g1.nfields);
    lsb::note_launch();
    k_helm_s<MT1, NC><<<grid, L::NT, L::smem, s>>>(g1, g2);
    return true;
}

// Large grids: 4 or 6 warps (registers: the intermediate block and half the output tiles stay
// live at two CTAs per SM), whichever leaves less idle in the last wave; a tuned width other
// than these keeps the two separate contractions.  k chunks of 32 where Kp allows
template <int MT1>
bool helm_pick(const GemmArgs& g1, const GemmArgs& g2, cudaStream_t s) {
    if (small_grid(g1)) {
        // 8, 16 or 32 columns per CTA: the least time on the busiest SM, a CTA taking as long as
        // its column groups and about two more for its loads (ties to the wider CTA)
        const long long nsm = sm_count();
        auto cost = [&](int nc) { return ((g1.C + 8 * nc - 1) / (8 * nc) * g1.nfields + nsm - 1) / nsm * (nc + 2); };
        const long long c4 = cost(4), c2 = cost(2), c1 = cost(1);
        if (c4 <= c2 && c4 <= c1) return helm_small_t<MT1, 4>(g1, g2, s);
        if (c2 <= c1) return helm_small_t<MT1, 2>(g1, g2, s);
        return helm_small_t<MT1, 1>(g1, g2, s);
    }
    constexpr int KC = (MT1 % 2 == 0) ? 32 : 16;
    int nw = helm_wave_eff<MT1, 4, KC>(g1) > helm_wave_eff<MT1, 6, KC>(g1) + 0.02 ? 4 : 6;
    if (g1.nw != 0) nw = g1.nw;
    if (nw == 4) return helm_launch_t<MT1, 4, KC>(g1, g2, s);
    if (nw == 6) return helm_launch_t<MT1, 6, KC>(g1, g2, s);
    return false;
}

bool launch_helm_fused(const GemmArgs& g1, const GemmArgs& g2, cudaStream_t s) {
    // the shapes the kernels assume: E^-1 and E square over the same padded k range, the rows
    // of E the interior rows of the solution
    if (g1.epi != EPI_HELM_SCALE || g2.epi != EPI_LIFT_ADD) return false;
    if (g1.Kp != g1.Mp || g2.Kp != g1.Mp || g2.Mp != g1.Mp || g2.M != g1.M || g2.K != g1.M) return false;
    if (g2.koff != 0 || g2.roff != 1 || g1.C != g2.C || g1.nfields != g2.nfields) return false;
    switch (g1.Mp / 16) {
        case 1: return helm_pick<1>(g1, g2, s);
        case 2: return helm_pick<2>(g1, g2, s);
        case 3: return helm_pick<3>(g1, g2, s);
        case 4: return helm_pick<4>(g1, g2, s);
        case 5: return helm_pick<5>(g1, g2, s);
        case 6: return helm_pick<6>(g1, g2, s);
        case 7: return helm_pick<7>(g1, g2, s);
        case 8: return helm_pick<8>(g1, g2, s);
        default: return false;  // nzm > 128: the intermediate does not fit the registers
    }
}

}  // namespace lsb
