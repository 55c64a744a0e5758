// The resident stepper's kernel (resident.cuh), a translation unit of its own.
#include <cuda_runtime.h>
#include "resident.cuh"
#include "tma.cuh"

namespace edus {

namespace {

__device__ __forceinline__ unsigned cluster_map(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_st(unsigned addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};\n" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void cluster_barrier(int CS) {
    if (CS == 1) {
        __syncthreads();
        return;
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// x / d by one multiplication, exact while x d < 2^32 (every index here)
struct Div32 {
    unsigned m;
    int d;
};
__device__ __forceinline__ Div32 make_div(int d) { return Div32{d > 1 ? (unsigned)(0x100000000ull / (unsigned)d) + 1u : 0u, d}; }
__device__ __forceinline__ int quot(int x, const Div32& f) { return f.m ? (int)__umulhi((unsigned)x, f.m) : x; }

// The twiddles w^d = exp(-+2 pi i a d / M) are root[d a tw_step] (a d < M, so
// inside the table), atw = a tw_step.
template <int R, bool FWD>
__device__ __forceinline__ void twiddle_all(double2* v, const double2* root, int atw) {
#pragma unroll
    for (int d = 1; d < R; ++d) {
        double2 w = root[d * atw];
        if (!FWD) w.y = -w.y;
        v[d] = cmul(v[d], w);
    }
}
template <int R, bool FWD>
__device__ __forceinline__ void butterfly_direct(double2* v, const double2* root, int atw, const ResStage& st) {
    const int n = st.n;
    if (FWD) {
        Dft<R, -1, double2>::run(v, root, n);
        if (st.tw) twiddle_all<R, true>(v, root, atw);
    } else {
        if (st.tw) twiddle_all<R, false>(v, root, atw);
        Dft<R, +1, double2>::run(v, root, n);
    }
}

// A stage over nbuf (1 or 2) buffers; table entry of task t: base | atw <<
// kResidentBase, element b of the butterfly at base + b step.  place(which, base)
// returns the butterfly's store, a callable (b, value).
template <int R, bool FWD, typename Place>
__device__ __forceinline__ void res_stage(const double2* buf, int nbuf, int bufstride, const ResStage& st,
                                          const unsigned* tt, const double2* rt, Place place) {
    for (int t = threadIdx.x; t < st.nt * nbuf; t += blockDim.x) {
        const int which = t >= st.nt;
        const unsigned e = tt[st.off + t - (which ? st.nt : 0)];
        const int base = e & ((1u << kResidentBase) - 1u);
        const double2* X = buf + (which ? bufstride : 0) + base;
        double2 v[R];
#pragma unroll
        for (int b = 0; b < R; ++b) v[b] = X[b * st.step];
        butterfly_direct<R, FWD>(v, rt + st.root, e >> kResidentBase, st);
        auto store = place(which, base);
#pragma unroll
        for (int b = 0; b < R; ++b) store(b, v[b]);
    }
}

// the stage's radix as a compile-time constant
template <int MASK, typename F>
__device__ __forceinline__ void with_radix(int r, F f) {
#define EDUS_RES_CASE(R)                        \
    case R:                                     \
        if constexpr ((MASK >> R) & 1) f(std::integral_constant<int, R>{}); \
        break;
    switch (r) {
        EDUS_RES_CASE(2)
        EDUS_RES_CASE(3)
        EDUS_RES_CASE(4)
        EDUS_RES_CASE(5)
        EDUS_RES_CASE(6)
        EDUS_RES_CASE(7)
        EDUS_RES_CASE(8)
        EDUS_RES_CASE(9)
        EDUS_RES_CASE(10)
        EDUS_RES_CASE(11)
        EDUS_RES_CASE(12)
        EDUS_RES_CASE(13)
    }
#undef EDUS_RES_CASE
}

}  // namespace

template <bool COUL, bool RK, int MASK>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_steps_kernel(ResidentArgs a, ResidentGeom g, const __grid_constant__ PlanePlan pl) {
    extern __shared__ double2 rsm[];
    const int Nk = a.Nk, nb = a.nb, P = nb * nb, CS = g.CS, RC = g.RC, NC = g.NC;
    const int N0 = pl.ax[0].n, N2 = pl.ax[2].n, N12 = Nk / N0;
    const int rank = blockIdx.x % CS, b = blockIdx.x / CS;
    const int KC = RC * N12, rows = P * KC;                 // local k points of every plane
    const int r0 = rank * RC, nr = min(RC, N0 - r0), nk = nr * N12, k0 = r0 * N12;
    const int c0 = rank * NC, ncol = max(0, min(NC, P * N12 - c0));
    // shared memory
    double2* XR = rsm;                                      // rows: stage input, then G
    double2* HR = XR + rows;                                // HSEX: the Hamiltonian
    double2* XC = HR + (COUL ? rows : 0);                   // columns
    double2* YC = XC + N0 * NC;
    double2* Rk = YC + (COUL ? N0 * NC : 0);                // stage input in k, two buffers when several tiles read one k
    const int Rd = nb > 2 ? rows : 0;
    double2* next = Rk + rows + Rd;
    const long long gb = (long long)b * a.S + k0;           // local element (p, k) of a global array: gb + p Nk + k
    const int pitch_s = KC;
    double2* Hm = g.h_smem ? next : a.ham + gb;             // H0 + E.xi
    next += g.h_smem ? rows : 0;
    double2* Ak = g.a_smem ? next : a.acc + gb;
    next += g.a_smem ? rows : 0;
    double2* Yk = g.y_smem ? next : a.y + gb;
    next += g.y_smem ? rows : 0;
    const int ph = g.h_smem ? pitch_s : Nk, pa = g.a_smem ? pitch_s : Nk, py = g.y_smem ? pitch_s : Nk;
    double2* rt = next;                                     // transform roots
    double2* hh = rt + a.ntab;                              // [nb] Hartree shifts
    double2* dg = hh + nb;                                  // [nb] rho_nn(R = 0)
    double* rq = (double*)(dg + nb);                        // coordinates
    unsigned* tt = (unsigned*)(rq + a.ntab + (a.ntab & 1)); // butterfly table
    ResStage(*sd)[kMaxStages] = (ResStage(*)[kMaxStages])(tt + g.ntt);  // stages per axis
    const int T = blockDim.x, tid = threadIdx.x;
    const Div32 fKC = make_div(KC), fN12 = make_div(N12), fNC = make_div(NC), fRC = make_div(RC), fN2 = make_div(N2);
    for (int i = tid; i < a.ntab; i += T) {
        rt[i] = __ldg(&a.roots[i]);
        rq[i] = __ldg(&a.rpos[i]);
    }
    // stages of axis 0 (columns), then of axes 1 and 2 (rows), and their tables
    {
        int off = 0;
        for (int d = 0; d < 3; ++d) {
            const AxisPlan& ax = pl.ax[d];
            const int inner = d == 0 ? NC : ax.inner, total = d == 0 ? N0 * NC : rows;
            for (int s = 0; s < ax.nst; ++s) {
                const int R = ax.r[s], L = ax.L[s], nbf = ax.n / R;
                if (tid == 0) sd[d][s] = ResStage{R, total / R, off, L * inner, ax.n, ax.rootoff, L > 1};
                for (int t = tid; t < total / R; t += T) {
                    const int in = t % inner, u = t / inner, o = u / nbf, bf = u - o * nbf, blk = bf / L, aa = bf - blk * L;
                    tt[off + t] = (unsigned)(o * ax.n * inner + in + (blk * L * R + aa) * inner) |
                                  ((unsigned)(aa * (ax.n / (L * R))) << kResidentBase);
                }
                off += total / R;
            }
        }
    }
    const double* rp0 = rq + pl.ax[0].rposoff;
    const double* rp1 = rq + pl.ax[1].rposoff;
    const double* rp2 = rq + pl.ax[2].rposoff;
    const unsigned xc_addr = smem_u32(XC), xr_addr = smem_u32(XR);
    // element (band pair and axes-1,2 position `col`, axis-0 index i0) to its column owner
    auto to_column = [&](int col, int i0, double2 v) {
        const int o = quot(col, fNC), off = i0 * NC + col - o * NC;
        if (CS == 1) XC[off] = v;
        else cluster_st(cluster_map(xc_addr + (unsigned)off * 16u, o), v);
    };
    const int nst0 = pl.ax[0].nst, nst1 = pl.ax[1].nst, nst2 = pl.ax[2].nst;
    cluster_barrier(CS);  // every CTA of the cluster runs, and the tables are written
    const bool flat = N12 == 1;  // no row transforms: the stage input goes straight to the columns
    for (int e = tid; e < rows; e += T) {
        const int p = quot(e, fKC), k = e - p * KC;
        if (k < nk) {
            const double2 v = a.y[gb + (long long)p * Nk + k];
            Rk[e] = v;
            if (g.y_smem) Yk[e] = v;
            if (flat) to_column(p, r0 + k, v);
            else XR[e] = v;
        } else {
            Rk[e] = XR[e] = make_double2(0.0, 0.0);
        }
    }
    int cur = 0;  // buffer of R holding the stage input
    const int half = (nb + 1) / 2, ntile = half * half;
    const Div32 fhalf = make_div(half);
    constexpr int NST = RK ? 4 : 1;
    StageField F = a.field[b];
    double lastE[3] = {0.0, 0.0, 0.0};
    bool haveH = false;
    if (flat) cluster_barrier(CS);
    else __syncthreads();

    for (int i = 0; i < a.steps; ++i) {
#pragma unroll 1
        for (int s = 0; s < NST; ++s) {
            // the next stage's field, requested a stage ahead
            const int nxt = i * NST + s + 1;
            const StageField Fn = a.field[(size_t)min(nxt, a.steps * NST - 1) * a.B + b];
            if (!haveH || F.E[0] != lastE[0] || F.E[1] != lastE[1] || F.E[2] != lastE[2]) {
                const long long mb = (long long)b * a.mstride + k0;
                const bool e0 = F.E[0] != 0.0, e1 = F.E[1] != 0.0, e2 = F.E[2] != 0.0;
                constexpr int U = 4;
                for (int e = tid; e < rows; e += U * T) {
                    double2 h[U], x0[U], x1[U], x2[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int eu = e + u * T, p = quot(eu, fKC), k = eu - p * KC;
                        const long long m = mb + (long long)p * Nk + k;
                        if (eu < rows && k < nk) {
                            h[u] = __ldg(&a.H0[m]);
                            if (e0) x0[u] = __ldg(&a.xi[0][m]);
                            if (e1) x1[u] = __ldg(&a.xi[1][m]);
                            if (e2) x2[u] = __ldg(&a.xi[2][m]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int eu = e + u * T, p = quot(eu, fKC), k = eu - p * KC;
                        if (eu >= rows || k >= nk) continue;
                        double2 v = h[u];
                        if (e0) { v.x += F.E[0] * x0[u].x; v.y += F.E[0] * x0[u].y; }
                        if (e1) { v.x += F.E[1] * x1[u].x; v.y += F.E[1] * x1[u].y; }
                        if (e2) { v.x += F.E[2] * x2[u].x; v.y += F.E[2] * x2[u].y; }
                        Hm[p * ph + k] = v;
                    }
                }
                haveH = true;
                lastE[0] = F.E[0];
                lastE[1] = F.E[1];
                lastE[2] = F.E[2];
            }
            // rows, k -> R (the last stage stores to the columns)
            if (!flat) {
                const int nrow = nst1 + nst2;
#pragma unroll 1
                for (int q = 0; q < nrow; ++q) {
                    const ResStage st = q < nst1 ? sd[1][q] : sd[2][q - nst1];
                    const bool out = q == nrow - 1;
                    with_radix<MASK>(st.r, [&](auto R) {
                        res_stage<R.value, true>(XR, 1, 0, st, tt, rt, [&](int, int base) {
                            // the butterfly's elements share their row
                            const int p = quot(base, fKC), k = base - p * KC, i = quot(k, fN12);
                            const int col = p * N12 + k - i * N12, i0 = r0 + i;
                            const bool live = i < nr;
                            return [=, &to_column](int b, double2 v) {
                                if (!out) XR[base + b * st.step] = v;
                                else if (live) to_column(col + b * st.step, i0, v);
                            };
                        });
                    });
                    if (!out) __syncthreads();
                }
                cluster_barrier(CS);
            }
            // columns: k -> R, pointwise, R -> k (the last stage stores to the rows)
            {
                const int tot = N0 * NC;
                // a column's elements to the row owners; `which` the Hamiltonian behind G
                auto to_rows = [&](int which, int base, int step0) {
                    const int i0 = quot(base, fNC), col = c0 + base - i0 * NC;
                    const int p = quot(col, fN12);
                    const int off = p * KC + col - p * N12 + (which ? rows : 0);
                    const bool live = col < P * N12;
                    return [=](int b, double2 v) {
                        const int i = i0 + b * step0, o = quot(i, fRC);
                        const int at = off + (i - o * RC) * N12;
                        if (CS == 1) XR[at] = v;
                        else if (live) cluster_st(cluster_map(xr_addr + (unsigned)at * 16u, o), v);
                    };
                };
                auto put_diag = [&](int n, double2 v) {  // rho_nn(R = 0), to every CTA
                    for (int o = 0; o < CS; ++o) cluster_st(cluster_map(smem_u32(&dg[n]), o), v);
                };
#pragma unroll 1
                for (int q = 0; q + 1 < nst0; ++q) {
                    const ResStage st = sd[0][q];
                    with_radix<MASK>(st.r, [&](auto R) {
                        res_stage<R.value, true>(XC, 1, 0, st, tt, rt, [&](int, int base) {
                            return [=](int b, double2 v) { XC[base + b * st.step] = v; };
                        });
                    });
                    __syncthreads();
                }
                if (nst0 > 0) {
                    const ResStage st = sd[0][nst0 - 1];
                    with_radix<MASK>(st.r, [&](auto RR) {
                        constexpr int R = RR.value;
                        for (int t = tid; t < st.nt; t += T) {
                            const unsigned en = tt[st.off + t];
                            const int base = en & ((1u << kResidentBase) - 1u);
                            const int q0 = quot(base, fNC), col = c0 + base - q0 * NC;
                            if (col >= P * N12) continue;
                            const int p = quot(col, fN12), q12 = col - p * N12, q1 = quot(q12, fN2), q2 = q12 - q1 * N2;
                            const double dot12 = F.g[1] * rp1[q1] + F.g[2] * rp2[q2];
                            const long long m = (long long)p * Nk + (long long)q0 * N12 + q12;
                            const double2* root = rt + st.root;
                            // the last stage's sub-length is 1: its butterfly's positions are consecutive
                            double2 v[R];
                            double w[COUL ? R : 1];
                            double2 z[COUL ? R : 1];
                            if (COUL) {
#pragma unroll
                                for (int q = 0; q < R; ++q) {
                                    z[COUL ? q : 0] = __ldg(&a.rho0p[m + q * N12]);
                                    w[COUL ? q : 0] = __ldg(&a.Wp[m + q * N12]);
                                }
                            }
#pragma unroll
                            for (int q = 0; q < R; ++q) v[q] = XC[base + q * st.step];
                            Dft<R, -1, double2>::run(v, root, st.n);
#pragma unroll
                            for (int q = 0; q < R; ++q) {
                                const double dot = F.g[0] * rp0[q0 + q] + dot12;
                                const double2 r = cscale(v[q], a.inv_nk);
                                v[q] = make_double2(-dot * r.y, dot * r.x);
                                if (COUL) {
                                    const double wq = w[COUL ? q : 0];
                                    // read back below by this thread (registers)
                                    YC[base + q * st.step] = make_double2(-wq * (r.x - z[COUL ? q : 0].x), -wq * (r.y - z[COUL ? q : 0].y));
                                    if (q == 0 && q0 == 0 && q12 == 0 && p % (nb + 1) == 0) put_diag(p / (nb + 1), r);
                                }
                            }
#pragma unroll 1
                            for (int which = 0; which < (COUL ? 2 : 1); ++which) {
                                if (which) {
#pragma unroll
                                    for (int q = 0; q < R; ++q) v[q] = YC[base + q * st.step];
                                }
                                Dft<R, +1, double2>::run(v, root, st.n);
                                if (nst0 == 1) {
                                    auto put = to_rows(which, base, 1);
#pragma unroll
                                    for (int q = 0; q < R; ++q) put(q, v[q]);
                                } else {
#pragma unroll
                                    for (int q = 0; q < R; ++q) XC[(which ? tot : 0) + base + q * st.step] = v[q];
                                }
                            }
                        }
                    });
                } else {
                    // one point on axis 0: the pointwise step alone
                    for (int e = tid; e < tot; e += T) {
                        const int col = c0 + e;
                        if (col >= P * N12) continue;
                        const int p = quot(col, fN12), q12 = col - p * N12, q1 = quot(q12, fN2), q2 = q12 - q1 * N2;
                        const double dot = F.g[0] * rp0[0] + F.g[1] * rp1[q1] + F.g[2] * rp2[q2];
                        const double2 r = cscale(XC[e], a.inv_nk);
                        to_rows(0, e, 1)(0, make_double2(-dot * r.y, dot * r.x));
                        if (COUL) {
                            const double2 z = __ldg(&a.rho0p[(long long)p * Nk + q12]);
                            const double w = __ldg(&a.Wp[(long long)p * Nk + q12]);
                            to_rows(1, e, 1)(0, make_double2(-w * (r.x - z.x), -w * (r.y - z.y)));
                            if (q12 == 0 && p % (nb + 1) == 0) put_diag(p / (nb + 1), r);
                        }
                    }
                }
                if (nst0 > 1) __syncthreads();
#pragma unroll 1
                for (int q = nst0 - 2; q >= 0; --q) {
                    const ResStage st = sd[0][q];
                    const int L = pl.ax[0].L[q];
                    with_radix<MASK>(st.r, [&](auto R) {
                        res_stage<R.value, false>(XC, COUL ? 2 : 1, tot, st, tt, rt, [&](int which, int base) {
                            auto put = to_rows(which, base, L);
                            return [=](int b, double2 v) {
                                if (q == 0) put(b, v);
                                else XC[(which ? tot : 0) + base + b * st.step] = v;
                            };
                        });
                    });
                    if (q > 0) __syncthreads();
                }
            }
            cluster_barrier(CS);
            // rows, R -> k; the Hamiltonian's last stage adds H0 + E.xi
            if (!flat) {
#pragma unroll 1
                for (int q = nst1 + nst2 - 1; q >= 0; --q) {
                    const ResStage st = q < nst1 ? sd[1][q] : sd[2][q - nst1];
                    with_radix<MASK>(st.r, [&](auto R) {
                        res_stage<R.value, false>(XR, COUL ? 2 : 1, rows, st, tt, rt, [&](int which, int base) {
                            const int p = quot(base, fKC), k = base - p * KC;
                            const bool add = COUL && which && q == 0 && k < nk;
                            const double2* hm = Hm + p * ph + k;
                            return [=](int b, double2 v) {
                                if (add) v = cadd(v, hm[b * st.step]);
                                XR[(which ? rows : 0) + base + b * st.step] = v;
                            };
                        });
                    });
                    __syncthreads();
                }
            } else if (COUL) {
                for (int e = tid; e < rows; e += T) {
                    const int p = quot(e, fKC), k = e - p * KC;
                    if (k < nk) HR[e] = cadd(HR[e], Hm[p * ph + k]);
                }
                __syncthreads();
            }
            if (COUL) {
                for (int n = tid; n < nb; n += T) {
                    double2 h = make_double2(0.0, 0.0);
                    for (int m = 0; m < nb; ++m)
                        h = cadd(h, cmul(__ldg(&a.hartree[n * nb + m]), csub(dg[m], __ldg(&a.rho0diag[m]))));
                    hh[n] = h;
                }
                __syncthreads();
            }
            const double2* R = Rk + cur * Rd;
            double2* Rn = Rk + (cur ^ 1) * Rd;
            const double2* H = COUL ? HR : Hm;
            const int pH = COUL ? KC : ph;
            const double ca = RK ? (s < 2 ? a.dt / 2. : (s == 2 ? a.dt : a.dt / 6.)) : 0.0;
            const double cb = RK ? (s == 0 ? a.dt / 6. : a.dt / 3.) : 0.0;
            for (int task = tid; task < ntile * KC; task += T) {
                const int tile = quot(task, fKC), k = task - tile * KC;
                if (k >= nk) continue;
                const int ti = quot(tile, fhalf);
                const int i0 = 2 * ti, j0 = 2 * (tile - ti * half);
                const int i1 = min(i0 + 1, nb - 1), j1 = min(j0 + 1, nb - 1);  // an odd band count repeats its last row
                double2 y[4], ac[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int p = ((q >> 1) ? i1 : i0) * nb + ((q & 1) ? j1 : j0);
                    if (!RK || s < 3) y[q] = Yk[p * py + k];
                    if (RK && s > 0) ac[q] = Ak[p * pa + k];
                }
                double2 c[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) c[q] = make_double2(0.0, 0.0);
#pragma unroll 2
                for (int l = 0; l < nb; ++l) {
                    const double2 h0 = H[(i0 * nb + l) * pH + k], h1 = H[(i1 * nb + l) * pH + k];
                    const double2 w0 = R[(l * nb + j0) * KC + k], w1 = R[(l * nb + j1) * KC + k];
                    const double2 q0 = R[(i0 * nb + l) * KC + k], q1 = R[(i1 * nb + l) * KC + k];
                    const double2 g0 = H[(l * nb + j0) * pH + k], g1 = H[(l * nb + j1) * pH + k];
                    auto mac = [](double2& z, double2 u, double2 v, double2 x, double2 w) {  // z += u v - x w
                        z.x = fma(u.x, v.x, fma(-u.y, v.y, z.x));
                        z.y = fma(u.x, v.y, fma(u.y, v.x, z.y));
                        z.x = fma(-x.x, w.x, fma(x.y, w.y, z.x));
                        z.y = fma(-x.x, w.y, fma(-x.y, w.x, z.y));
                    };
                    mac(c[0], h0, w0, q0, g0);
                    mac(c[1], h0, w1, q0, g1);
                    mac(c[2], h1, w0, q1, g0);
                    mac(c[3], h1, w1, q1, g1);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int n = i0 + (q >> 1), m = j0 + (q & 1);
                    if (n >= nb || m >= nb) continue;
                    const int p = n * nb + m, e = p * KC + k;
                    if (COUL) c[q] = cadd(c[q], cmul(csub(hh[n], hh[m]), R[e]));
                    const double2 G = XR[e];
                    const double2 f = make_double2(G.x + c[q].y, G.y - c[q].x);
                    double2 out;
                    if (RK) {
                        if (s < 3) {
                            out = make_double2(y[q].x + ca * f.x, y[q].y + ca * f.y);
                            const double2 z = s == 0 ? y[q] : ac[q];
                            Ak[p * pa + k] = make_double2(z.x + cb * f.x, z.y + cb * f.y);
                        } else {
                            out = make_double2(ac[q].x + ca * f.x, ac[q].y + ca * f.y);
                            Yk[p * py + k] = out;
                        }
                    } else {
                        const long long ge = gb + (long long)p * Nk + k;
                        const int ph0 = i % a.order;  // the ring's rotation since the first step
                        double2 hq[5];
#pragma unroll
                        for (int o = 1; o < 5; ++o)
                            if (o < a.order) hq[o] = a.hist[o >= ph0 ? o - ph0 : o - ph0 + a.order][ge];
                        out = make_double2(y[q].x + a.c[0] * f.x, y[q].y + a.c[0] * f.y);
#pragma unroll
                        for (int o = 1; o < 5; ++o)
                            if (o < a.order) out = make_double2(out.x + a.c[o] * hq[o].x, out.y + a.c[o] * hq[o].y);
                        a.hist[ph0 ? a.order - ph0 : 0][ge] = f;
                        Yk[p * py + k] = out;
                    }
                    Rn[e] = out;
                    if (flat) to_column(p, r0 + k, out);
                    else XR[e] = out;
                }
            }
            cur ^= Rd ? 1 : 0;
            F = Fn;
            if (flat) cluster_barrier(CS);
            else __syncthreads();
        }
    }
    if (g.y_smem)
        for (int e = tid; e < rows; e += T) {
            const int p = quot(e, fKC), k = e - p * KC;
            if (k < nk) a.y[gb + (long long)p * Nk + k] = Yk[e];
        }
    cluster_barrier(CS);
}

ResidentKernel resident_kernel(bool coul, bool rk, bool all) {
    if (coul) {
        if (rk) return all ? resident_steps_kernel<true, true, kRadixAll> : resident_steps_kernel<true, true, kRadixCommon>;
        return all ? resident_steps_kernel<true, false, kRadixAll> : resident_steps_kernel<true, false, kRadixCommon>;
    }
    if (rk) return all ? resident_steps_kernel<false, true, kRadixAll> : resident_steps_kernel<false, true, kRadixCommon>;
    return all ? resident_steps_kernel<false, false, kRadixAll> : resident_steps_kernel<false, false, kRadixCommon>;
}

}  // namespace edus
