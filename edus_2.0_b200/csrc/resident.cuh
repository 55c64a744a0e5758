// Whole propagations of small problems in one launch: a cluster of CTAs holds
// a solve in its shared memory and runs every RK4 or Adams-Bashforth step of
// the call, so a stage costs two cluster barriers instead of two to four
// kernel launches.
//
// What bounds such a problem is latency: a stage of the two-band chain (64 k
// points) moves 4 KB and took 8.5 us as two launches, 4.6 us here; of two bands
// on 50 x 50 about 22 us as four launches, 11 us here; with HSEX on 40 x 40 26 us
// and 12 us.
//
// Split (grid N0 x N12, N12 = N1 N2).  CTA r owns RC rows of axis 0 of every
// band pair: it transforms them along axes 1 and 2 and does everything that is
// local in k (commutator, stage update, Hamiltonian).  The transform along axis
// 0 runs on columns: the P N12 columns (band pair, position on axes 1, 2) are
// dealt to the CTAs in equal runs.  Two exchanges a stage, both by stores into
// the owner's shared memory from the registers of the butterfly that produces
// the value, so that no pass over shared memory and no remote read's latency is
// added:
//   rows: k -> R on axes 1, 2 | store to the column owners, cluster barrier |
//   columns: k -> R on axis 0; the last stage, the pointwise step and the first
//     inverse stage are one pass in registers; R -> k on axis 0
//   | store to the row owners, cluster barrier |
//   rows: R -> k on axes 1, 2; C = H rho - rho H on 2 x 2 tiles of one k point,
//     f = G - i C, stage update; the new stage input replaces G in place.
// H0 + E.xi is rebuilt only when E changed from the stage before (stages 2 and
// 3 of RK4 share their time, as do stage 4 and the next step's first).  Butterfly
// addresses and twiddle indices come from a table made once per launch, and the
// twiddles from the root table instead of by powers: here latency, not shared
// memory bandwidth, is scarce.
// Reference: Functional_SourceTerm.hpp:15-50, DESolver.hpp:154-220.
#pragma once
#include <algorithm>
#include "fft_plane.cuh"
#include "stage_field.hpp"

namespace edus {

struct ResidentArgs {
    const double2* H0;     // [P][Nk] (+ mstride per solve)
    const double2* xi[3];
    long long mstride;
    const double2* rho0p;  // HSEX: model planes in digit-reversed R order
    const double* Wp;
    const double2* hartree;
    const double2* rho0diag;
    double2* y;            // [B][P][Nk]: read at the start, written at the end
    double2* acc;          // RK accumulator and model Hamiltonian, [B][P][Nk], where
    double2* ham;          //   shared memory has no room for them
    double2* hist[5];      // AB: in ring order at the first step
    double c[5];           // AB: dt beta
    int order;
    const StageField* field;  // [steps][stages][B]
    int steps, B;
    const double2* roots;
    const double* rpos;
    int ntab;              // entries of either table
    long long S;
    int Nk, nb;
    double inv_nk, dt;
};

struct ResidentGeom {
    int CS, RC, NC, threads;
    int ntt;          // entries of the butterfly table
    int y_smem, a_smem, h_smem;  // Y, A, H0 + E.xi in shared memory
    size_t smem;
};

constexpr int kResidentThreads = 384;  // 168 registers a thread
constexpr int kResidentBase = 18;  // bits of a table entry that hold the butterfly's base address

// One stage of the CTA's lines along an axis: butterflies, table offset, element
// step of a butterfly, twiddle roots, whether there are twiddles (not in an
// axis's last stage, whose sub-length is 1).
struct ResStage {
    int r, nt, off, step, n, root, tw;
};

// Geometry for clusters of at most cs CTAs; smem 0 if it does not fit `limit`.
inline ResidentGeom resident_geometry(const PlanePlan& pl, int nb, bool coul, bool rk, int cs, int ntab, size_t limit) {
    ResidentGeom g{};
    const int P = nb * nb, N0 = pl.ax[0].n, N12 = pl.Nk / N0;
    g.RC = (N0 + cs - 1) / cs;
    g.CS = (N0 + g.RC - 1) / g.RC;
    g.NC = (P * N12 + g.CS - 1) / g.CS;
    const size_t rows = (size_t)P * g.RC * N12, cols = (size_t)N0 * g.NC;
    if (rows >= (1u << kResidentBase) || cols >= (1u << kResidentBase)) return g;
    int tasks = ((nb + 1) / 2) * ((nb + 1) / 2) * g.RC * N12;
    for (int d = 0; d < 3; ++d)
        for (int s = 0; s < pl.ax[d].nst; ++s) {
            const size_t t = (d == 0 ? cols : rows) / pl.ax[d].r[s];
            g.ntt += (int)t;
            tasks = std::max(tasks, (int)t);
        }
    g.threads = std::min(kResidentThreads, std::max(64, (tasks + 31) & ~31));
    size_t need = (rows * (1 + (nb > 2 ? 2 : 1) + (coul ? 1 : 0)) + cols * (coul ? 2 : 1) + ntab + (ntab + 1) / 2 +
                   2 * nb + (g.ntt + 3) / 4) * 16 +
                  ((3 * kMaxStages * sizeof(ResStage) + 15) & ~(size_t)15);
    if (need > limit) return g;
    auto room = [&]() {
        if (need + rows * 16 > limit) return 0;
        need += rows * 16;
        return 1;
    };
    g.h_smem = room();
    g.a_smem = rk ? room() : 0;
    g.y_smem = room();
    g.smem = need;
    return g;
}

using ResidentKernel = void (*)(ResidentArgs, ResidentGeom, PlanePlan);
// the kernel of a form (all: radices 11 and 13 compiled in)
ResidentKernel resident_kernel(bool coul, bool rk, bool all);

}  // namespace edus
