// Batched banded solves of the Laplacian / Helmholtz operators, FP64.
//
// Restates the per-(m,k) systems of mod_legops.f90 IDEL2LN (1013-1176),
// IDEL2 (823-1010) and IHELM (1204-1354), factored without pivoting as
// LUDCMPB/LUBKSBB do (mod_bandmat.f90:65-155, 320-401).  One thread owns one
// (m, k) system: it builds each band row on the fly from the DEL2H/XM
// coefficient tables, eliminates its sub-diagonal entries against the
// previous pivot rows (kept in registers), writes the resulting U row to a
// scratch array laid out [row][entry][system] (coalesced across threads),
// and back-substitutes in place.  Band entries that reach past the system's
// size are dropped, which is BANDAUX's truncation of each leading block.
//
//  kind 0  IDEL2LN: m = 0 systems carry the log-term column (k = 0), 5-band
//  kind 1  IDEL2:   m = 0 uses the 7-band row-shifted system (k = 0: row 0 is
//                   the log-term boundary condition)
//  kind 2  IHELM:   m = 0 solves (H XM) y = rhs on NN-1 rows, A = XM y
#include "bulk.cuh"
#include "mlegs_internal.h"
#include "project_tail.cuh"

#include <algorithm>

namespace mlegs {

namespace {
constexpr int MAXW = 7;  // band width bound (7-band m = 0 systems)
constexpr int RB = 6;    // rows whose loads are issued together; a multiple of 3 so that
                         // the 3-row pivot window is indexed by compile-time constants
}

struct BandRowCtx {
    const double* del2h;  // [NB][5] for this m
    const double* xm;     // [NB][2] for this m (m = 0 only)
    double shift;         // k^2 + alpha
    int kind, m, k;
    double l0, l1, l2;    // log-term column entries (IDEL2LN / IDEL2 at m = k = 0)
};

// Entry (row, col) of the original DEL2H - shift operator (with the log column).
__device__ __forceinline__ double del2_entry(const BandRowCtx& c, int row, int col) {
    int d = col - row;
    if (d < -2 || d > 2 || row < 0 || col < 0) return 0.0;
    double v = c.del2h[(size_t)row * 5 + (d + 2)];
    if (d == 0) v -= c.shift;
    if (col == 0 && (c.kind == 0 || c.kind == 1) && c.m == 0 && c.k == 0) {
        if (row == 0) v += c.l0;
        else if (row == 1) v += c.l1;
        else if (row == 2) v += c.l2;
    }
    return v;
}

// Row `row` of the system matrix, as entries at columns row-3..row+3 (w[0..6]).
__device__ __forceinline__ void build_row(const BandRowCtx& c, int row, double* w) {
#pragma unroll
    for (int q = 0; q < MAXW; ++q) w[q] = 0.0;
    if (c.m != 0 || c.kind == 0) {
        for (int d = -2; d <= 2; ++d) w[d + 3] = del2_entry(c, row, row + d);
        return;
    }
    if (c.kind == 1) {
        if (c.k != 0) {
            for (int d = -2; d <= 2; ++d) w[d + 3] = del2_entry(c, row, row + d);
        } else if (row == 0) {
            w[3] = 1.0;
        } else {
            // new row r = original row r-1 over the same columns
            for (int col = row - 3; col <= row + 1; ++col)
                if (col >= 0) w[col - row + 3] = del2_entry(c, row - 1, col);
        }
        return;
    }
    // kind 2, m = 0: (H XM)(row, col) = sum_l H(row, l) XM(l, col)
    for (int l = row - 2; l <= row + 2; ++l) {
        if (l < 0) continue;
        double h = del2_entry(c, row, l);
        if (h == 0.0) continue;
        const double* x = c.xm + (size_t)l * 2;
        // XM(l, l-1) = sub(l), XM(l, l) = 1, XM(l, l+1) = super(l)
        if (l - 1 >= 0) w[(l - 1) - row + 3] += h * x[0];
        w[l - row + 3] += h;
        w[(l + 1) - row + 3] += h * x[1];
    }
}

__global__ void solve_kernel(DevGrid g, double2* A, double* ln_out, int kind, double alp, int has_ln,
                             double ln_in, const double* b_ln, double* scratch, int pad) {
    const int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsys) return;
    const int k = t % g.NXCHOPDIM;
    const int m = t / g.NXCHOPDIM;
    int nn = g.NRCHOP + pad - m;
    if (nn < 0) nn = 0;
    BandRowCtx c;
    c.del2h = g.del2h + (size_t)m * g.NB * 5;
    c.xm = g.xm + (size_t)m * g.NB * 2;
    c.shift = g.ak[k] * g.ak[k] + ((kind == 2) ? alp : 0.0);
    c.kind = kind;
    c.m = m;
    c.k = k;
    c.l0 = 4.0 / 3 / g.ELL2;
    c.l1 = -2 * g.norm0[0] / g.norm0[1] / g.ELL2;
    c.l2 = 2.0 / 3 * g.norm0[0] / g.norm0[2] / g.ELL2;
    int lo = 2, up = 2;
    if (m == 0 && kind != 0) {
        lo = 3;
        up = 3;
    }
    int size = (m == 0 && kind == 2) ? nn - 1 : nn;
    double2* col = A + (size_t)m * g.NRCHOPDIM * g.NXCHOPDIM + k;
    const size_t st = g.NXCHOPDIM;
    if (size <= 0) return;
    // IDEL2 (m = 0, k = 0): shift the rhs down one row, row 0 <- LN BC (929-936)
    if (kind == 1 && m == 0 && k == 0) {
        for (int r = size - 1; r >= 1; --r) col[(size_t)r * st] = col[(size_t)(r - 1) * st];
        col[0] = make_double2(has_ln ? ln_in / g.norm0[0] : 0.0, 0.0);
    }
    // forward elimination; window of the last 3 pivot rows (U entries d = 0..up)
    double U[3][4];
    double2 R[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        R[a] = make_double2(0.0, 0.0);
#pragma unroll
        for (int b = 0; b < 4; ++b) U[a][b] = 0.0;
    }
    for (int r0 = 0; r0 < size; r0 += RB) {
        // each row reads only its own right-hand side, so the block's loads go first
        double2 rb[RB];
#pragma unroll
        for (int q = 0; q < RB; ++q) rb[q] = (r0 + q < size) ? col[(size_t)(r0 + q) * st] : make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            const int r = r0 + q;  // r0 is a multiple of 3: r % 3 == q % 3
            if (r >= size) break;
            double w[MAXW];
            build_row(c, r, w);
            double2 rhs = rb[q];
            // eliminate columns r-lo .. r-1 (left to right)
#pragma unroll
            for (int d = 3; d >= 1; --d) {
                if (d > lo || r - d < 0) continue;
                const int wi = (q - d + 3) % 3;  // (r - d) % 3
                const double f = w[3 - d] / U[wi][0];
                w[3 - d] = 0.0;
#pragma unroll
                for (int j = 1; j <= 3; ++j) {
                    if (j > up) continue;
                    const int qq = 3 - d + j;
                    if (qq < MAXW) w[qq] -= f * U[wi][j];
                }
                rhs.x -= f * R[wi].x;
                rhs.y -= f * R[wi].y;
            }
            const int wr = q % 3;
            U[wr][0] = w[3];
#pragma unroll
            for (int j = 1; j <= 3; ++j) U[wr][j] = (j <= up) ? w[3 + j] : 0.0;
            R[wr] = rhs;
#pragma unroll
            for (int j = 0; j <= 3; ++j) scratch[((size_t)r * 4 + j) * nsys + t] = U[wr][j];
            col[(size_t)r * st] = rhs;
        }
    }
    // back substitution
    double2 x1 = make_double2(0.0, 0.0), x2 = x1, x3 = x1;  // x[r+1], x[r+2], x[r+3]
    for (int r1 = size - 1; r1 >= 0; r1 -= RB) {
        double2 vb[RB];
        double ub[RB][4];
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            const int r = r1 - q;
            vb[q] = make_double2(0.0, 0.0);
            ub[q][0] = 1.0;
            ub[q][1] = ub[q][2] = ub[q][3] = 0.0;
            if (r >= 0) {
                vb[q] = col[(size_t)r * st];
#pragma unroll
                for (int j = 0; j < 4; ++j) ub[q][j] = scratch[((size_t)r * 4 + j) * nsys + t];
            }
        }
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            const int r = r1 - q;
            if (r < 0) break;
            double2 v = vb[q];
            const double u0 = ub[q][0], u1 = ub[q][1], u2 = ub[q][2], u3 = ub[q][3];
            if (r + 1 < size) { v.x -= u1 * x1.x; v.y -= u1 * x1.y; }
            if (r + 2 < size) { v.x -= u2 * x2.x; v.y -= u2 * x2.y; }
            if (r + 3 < size) { v.x -= u3 * x3.x; v.y -= u3 * x3.y; }
            v.x /= u0;
            v.y /= u0;
            col[(size_t)r * st] = v;
            x3 = x2;
            x2 = x1;
            x1 = v;
        }
    }
    if (m == 0 && kind == 2) {
        // A(NN) = 0; A(:NN) = XM(:NN) y  (1310-1316)
        col[(size_t)(nn - 1) * st] = make_double2(0.0, 0.0);
        double2 prev = make_double2(0.0, 0.0);
        for (int r = 0; r < nn; ++r) {
            double2 cur = col[(size_t)r * st];
            double2 nxt = (r + 1 < nn) ? col[(size_t)(r + 1) * st] : make_double2(0.0, 0.0);
            const double* x = c.xm + (size_t)r * 2;
            double2 v = cur;
            if (r >= 1) { v.x += x[0] * prev.x; v.y += x[0] * prev.y; }
            if (r + 1 < nn) { v.x += x[1] * nxt.x; v.y += x[1] * nxt.y; }
            col[(size_t)r * st] = v;
            prev = cur;
        }
    }
    if (m == 0 && k == 0) {
        if (kind == 0) {
            *ln_out = col[0].x * g.norm0[0];
            col[0] = make_double2(0.0, 0.0);
        } else if (kind == 1 && has_ln) {
            *ln_out = col[0].x * g.norm0[0];
        }
    }
}

// ---------------------------------------------------------------------------
// Factor once, solve many.  For a fixed (kind, pad, alp) the system matrices
// do not change from call to call, so their LU factors (the same unpivoted
// elimination as solve_kernel, LUDCMPB of mod_bandmat.f90:65-155) are stored
// once and every later solve is only the substitutions of LUBKSBB (320-401).
// The table holds blocks of 16 systems of one m (consecutive k), per row the
// sub-diagonal multipliers f_d = L(r, r-d) and the scaled U row u_d =
// U(r, r+d)/U(r, r), ri = 1/U(r, r) (formed here, off the substitution's
// recurrence), the 16 systems side by side and the entries in pairs for 16-byte loads:
//   5-band, HB = 2: L5 [block][row] {f2, f1}[16], U5 [block][row] {u2, u1}[16] ri[16],
//     block = (m, k / 16);
//   7-band m = 0 systems of kinds 1 and 2, HB = 3: L7 [k / 16][row] {f3, f2}[16] f1[16],
//     U7 [k / 16][row] {u3, u2}[16] {u1, ri}[16];
// so a run of rows is one contiguous piece, one bulk copy.
struct FactorTable {
    size_t u5, l7, u7, total;  // offsets (doubles); L5 starts at 0
    int nkb, R;                // blocks per m, rows per block
    __host__ __device__ explicit FactorTable(const DevGrid& g) {
        nkb = (g.NXCHOPDIM + 15) / 16;
        R = g.NRCHOPDIM;
        const size_t b = (size_t)nkb * R;
        u5 = g.NTCHOPDIM * b * 32;
        l7 = u5 + g.NTCHOPDIM * b * 48;
        u7 = l7 + b * 48;
        total = u7 + b * 64;
    }
};

__global__ void factor_kernel(DevGrid g, int kind, double alp, int pad, double* F) {
    const FactorTable ft(g);
    const int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsys) return;
    const int k = t % g.NXCHOPDIM;
    const int m = t / g.NXCHOPDIM;
    int nn = g.NRCHOP + pad - m;
    if (nn < 0) nn = 0;
    BandRowCtx c;
    c.del2h = g.del2h + (size_t)m * g.NB * 5;
    c.xm = g.xm + (size_t)m * g.NB * 2;
    c.shift = g.ak[k] * g.ak[k] + ((kind == 2) ? alp : 0.0);
    c.kind = kind;
    c.m = m;
    c.k = k;
    c.l0 = 4.0 / 3 / g.ELL2;
    c.l1 = -2 * g.norm0[0] / g.norm0[1] / g.ELL2;
    c.l2 = 2.0 / 3 * g.norm0[0] / g.norm0[2] / g.ELL2;
    const bool wide = (m == 0 && kind != 0);
    const int lo = wide ? 3 : 2, up = wide ? 3 : 2;
    const int size = (m == 0 && kind == 2) ? nn - 1 : nn;
    const size_t blk = wide ? (size_t)(k / 16) : (size_t)m * ft.nkb + k / 16;
    double* L = F + (wide ? ft.l7 : 0) + blk * ft.R * (wide ? 48 : 32);
    double* UU = F + (wide ? ft.u7 : ft.u5) + blk * ft.R * (wide ? 64 : 48);
    const int sy = k % 16;
    double U[3][4] = {};
    for (int r = 0; r < size; ++r) {
        double w[MAXW];
        build_row(c, r, w);
        double f[4] = {0.0, 0.0, 0.0, 0.0};
        for (int d = 3; d >= 1; --d) {
            if (d > lo || r - d < 0) continue;
            const int wi = (r - d) % 3;
            f[d] = w[3 - d] / U[wi][0];
            w[3 - d] = 0.0;
            for (int j = 1; j <= 3; ++j) {
                if (j > up) continue;
                const int qq = 3 - d + j;
                if (qq < MAXW) w[qq] -= f[d] * U[wi][j];
            }
        }
        const int wr = r % 3;
        U[wr][0] = w[3];
        for (int j = 1; j <= 3; ++j) U[wr][j] = (j <= up) ? w[3 + j] : 0.0;
        const double ri = 1.0 / w[3];
        double u[4];
        for (int j = 1; j <= up; ++j) u[j] = (r + j < size) ? __dmul_rn(U[wr][j], ri) : 0.0;
        double* l = L + (size_t)r * lo * 16;
        double* o = UU + (size_t)r * (up + 1) * 16;
        l[2 * sy] = f[lo];
        l[2 * sy + 1] = f[lo - 1];
        o[2 * sy] = u[up];
        o[2 * sy + 1] = u[up - 1];
        if (wide) {
            l[32 + sy] = f[1];
            o[32 + 2 * sy] = u[1];
            o[32 + 2 * sy + 1] = ri;
        } else {
            o[32 + sy] = ri;
        }
    }
}

size_t solve_factor_doubles(const DevGrid& g) { return FactorTable(g).total; }

// F: solve_factor_doubles(g) entries.
void k_solve_factor(const DevGrid& g, int kind, double alp, int pad, double* F, cudaStream_t s) {
    cudaMemsetAsync(F, 0, solve_factor_doubles(g) * sizeof(double), s);  // the blocks' unused columns
    const int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    factor_kernel<<<(nsys + 63) / 64, 64, 0, s>>>(g, kind, alp, pad, F);
    count_launch();
}

// The substitutions: a CTA takes a block of 16 systems.  Warp 0 runs them (lane =
// system x real or imaginary part); warp 1 streams the factor rows through a
// ring of SNST chunks of SCH rows in shared memory, ascending for the first
// substitution and descending for the second, and the right-hand sides with
// the first pass's chunks.  The column stays in shared memory until both warps
// write the solution.
//
// What bounds it: a system is a serial chain of rows and its warp runs alone,
// several cycles an instruction, so the launch lasts as long as the
// instructions of the longest (m = 0) blocks.  Hence the second warp for the
// copies, one bulk copy a chunk for the factors, the chunk's values in
// registers before the recurrence (then one dependent FMA per row), and the
// tables of the m = 0 tails (CALCAT1, XM) in shared memory.  IDEL2 and IDEL2LN at
// 192x128x256 (139 MB each) take 31 us; 51 us with each thread reading its rows 16
// at a time from global memory, 34 us with one warp doing both jobs.  A 58-row
// solve at 64x32x32 takes 11.6 us, 17-19 us in the other forms (ncu, cold cache).
// The blocks run m ascending: longest first.
// XG: columns too long for shared memory (NRCHOP + pad > 727 rows at SOLVE_SMEM_MAX)
// stay in global memory, read and written a chunk at a time, and so do the tables: its
// shared memory is the ring alone, for any number of rows.
namespace {
using namespace bulk;

constexpr int SCH = 8;   // rows per chunk
constexpr int SNST = 5;  // chunks in the ring
constexpr int SRING = SNST * SCH * 64;  // doubles

struct SolveForm {
    int kind, has_ln;
    double ln_in;
    int pad, farfield;
    int keep_tail;  // transposed systems: rows from the system size on are not written
};
// A block's shared memory: the ring, the tables of the m = 0 tails (at1 [R],
// xm [R][2]), the column Xs [R][16].
struct SolveShared {
    double* ring;
    const double* at1;
    const double* xm;
    double2* Xs;
    uint64_t* full;   // a chunk has arrived: 32 producer lanes and the bulk copy
    uint64_t* empty;  // the consumer has read it
    uint64_t* whole;  // the staged column of the transposed m = 0 system
    uint64_t limit;   // of the two warps' waits (0: WAIT_CYCLES)
};

// A whole warp's wait; false for all lanes when it runs out.  The warp then stops; the
// other one, which gets no more chunks or no more room, stops at its own next wait.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, int phase, const SolveShared& sh) {
    return __all_sync(0xffffffffu, bar_wait(bar, (uint32_t)(phase & 1), sh.limit));
}

// The stage back to the producing warp, whose next bulk copy writes over it through the
// async proxy: every lane's reads, which may still be in flight here (their values are used
// further down), come before that by the fence (1% of ten AB2-CN steps at 64x32x32).
__device__ __forceinline__ void give_back(uint64_t* empty) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) bar_arrive(empty);
}

// Chunk c of 2 nch: rows [lo, lo + rows), ascending in the first pass, descending in the second.
__device__ __forceinline__ void solve_chunk(int c, int nch, int size, int& lo, int& rows) {
    if (c < nch) {
        lo = c * SCH;
        rows = min(SCH, size - lo);
    } else {
        const int hi = size - (c - nch) * SCH;
        lo = max(0, hi - SCH);
        rows = hi - lo;
    }
}

// Returns the chunks issued: fewer than 2 nch when a wait ran out.
template <int HB, bool TR, bool XG>
__device__ int solve_producer(const DevGrid& g, const double2* src, int nsb, const double* FL, const double* FU,
                               int size, int nn, const SolveShared& sh) {
    constexpr int WL = HB * 16, WU = (HB + 1) * 16, WA = TR ? WU : WL, WB = TR ? WL : WU;
    const int lane = threadIdx.x & 31;
    const size_t NK = g.NXCHOPDIM;
    const int nch = (size + SCH - 1) / SCH;
    const int q = lane & 15, r0 = lane >> 4;
    const bool staged = TR && HB == 3;
    if (staged && !XG) {
        if (q < nsb)
            for (int r = r0; r < nn; r += 2) copy16_async(sh.Xs + r * 16 + q, src + (size_t)r * NK + q);
        copy16_arrive(sh.whole);
    }
    int c = 0;
    for (; c < 2 * nch; ++c) {
        const int st = c % SNST;
        if (c >= SNST && !warp_wait(sh.empty + st, c / SNST - 1, sh)) break;
        int lo, rows;
        solve_chunk(c, nch, size, lo, rows);
        const bool up = c < nch;
        const uint32_t fb = (uint32_t)(rows * (up ? WA : WB)) * 8u;
        if (lane == 0) {
            bar_expect_tx(sh.full + st, fb);
            bulk_copy(sh.ring + st * (SCH * 64), ((up != TR) ? FL : FU) + (size_t)lo * (up ? WA : WB), fb, sh.full + st);
        }
        if (up && !XG && !staged && q < nsb) {
#pragma unroll
            for (int i = 0; i < SCH / 2; ++i) {
                const int r = lo + r0 + 2 * i;
                if (r < lo + rows) copy16_async(sh.Xs + r * 16 + q, src + (size_t)r * NK + q);
            }
        }
        copy16_arrive(sh.full + st);
    }
    return c;
}

// After a wait ran out, in the producing warp: its copies in flight land (bounded waits
// again, at the full limit) before the CTA ends and its shared memory is another's.
__device__ void solve_drain(int issued, const SolveShared& sh) {
    for (int b = max(0, issued - SNST); b < issued; ++b) bar_wait(sh.full + b % SNST, (uint32_t)((b / SNST) & 1));
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// HB: half-bandwidth; TR: the transposed system U^T z = y, L^T x = z, else
// L y = b, U x = y with the tails.
// Returns the rows to write, -1 when a wait ran out.
template <int HB, bool TR, bool XG>
__device__ int solve_consumer(const DevGrid& g, const SolveItem& p, const SolveForm& fo, int m, int k0, int nsb,
                              int size, int nn, const SolveShared& sh) {
    const int lane = threadIdx.x, sy = lane >> 1, comp = lane & 1, k = k0 + sy;
    const size_t NK = g.NXCHOPDIM, st = 2 * NK, base = (size_t)m * g.NRCHOPDIM * NK + k0;
    const bool live = sy < nsb;
    const int kind = fo.kind;
    const int nch = (size + SCH - 1) / SCH;
    const double* sc = (const double*)(p.src + base + sy) + comp;
    double* dc = (double*)(p.dst + base + sy) + comp;
    double* X = (double*)sh.Xs + lane;
    const bool c00 = m == 0 && k == 0;
    constexpr int WL = HB * 16, WU = (HB + 1) * 16;  // doubles per row of L and U
    // a row's factors from the ring: f[d] = L(r, r-d), or f[0] = 1/U(r, r), f[d] = u_d
    auto row_l = [&](const double* row, double (&f)[HB + 1]) {
        const double2 a = *(const double2*)(row + 2 * sy);
        f[HB] = a.x;
        f[HB - 1] = a.y;
        if constexpr (HB == 3) f[1] = row[32 + sy];
    };
    auto row_u = [&](const double* row, double (&f)[HB + 1]) {
        const double2 a = *(const double2*)(row + 2 * sy);
        f[HB] = a.x;
        f[HB - 1] = a.y;
        if constexpr (HB == 3) {
            const double2 b = *(const double2*)(row + 32 + 2 * sy);
            f[1] = b.x;
            f[0] = b.y;
        } else {
            f[0] = row[32 + sy];
        }
    };
    auto xget = [&](int r) -> double { return XG ? (live ? dc[(size_t)r * st] : 0.0) : X[r * 32]; };
    auto xput = [&](int r, double v) {
        if (!XG) X[r * 32] = v;
        else if (live) dc[(size_t)r * st] = v;
    };
    // column <- A column for a tri-diagonal A of unit diagonal over rows < nn (XM and XM^T);
    // XM^T comes first and takes the right-hand side, which XG reads from src (src may be
    // dst: a row is read before its chunk is written)
    auto xm_pass = [&](bool transposed) {
        auto get = [&](int r) -> double {
            return XG && transposed ? (live ? sc[(size_t)r * st] : 0.0) : xget(r);
        };
        double prev = 0.0, cur = nn > 0 ? get(0) : 0.0;
        for (int r0 = 0; r0 < nn; r0 += SCH) {
            double nx[SCH], lo[SCH], hi[SCH];
#pragma unroll
            for (int q = 0; q < SCH; ++q) {
                const int r = r0 + q, rl = transposed ? r - 1 : r, rh = transposed ? r + 1 : r;
                const bool a = r >= 1 && r < nn, b = r + 1 < nn;
                nx[q] = b ? get(r + 1) : 0.0;
                lo[q] = a ? sh.xm[2 * rl + (transposed ? 1 : 0)] : 0.0;
                hi[q] = b ? sh.xm[2 * rh + (transposed ? 0 : 1)] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < SCH; ++q) {
                const int r = r0 + q;
                if (r >= nn) break;
                // explicit roundings: every launch form gives the same bits
                double v = transposed ? __fma_rn(lo[q], prev, __fma_rn(hi[q], nx[q], cur))
                                      : __fma_rn(hi[q], nx[q], __fma_rn(lo[q], prev, cur));
                xput(r, v);
                prev = cur;
                cur = nx[q];
            }
        }
    };
    // the transposed IHELM system at m = 0 takes w = XM^T y, which couples
    // neighbouring rows: the column is formed (nn rows, in dst for XG) before the passes
    constexpr bool staged = TR && HB == 3;
    if constexpr (staged) {
        if (!XG && !warp_wait(sh.whole, 0, sh)) return -1;
        xm_pass(true);
    }
    // IHELM of a right-hand side with a log term (mod_legops.f90:1244-1255)
    double lnv = 0.0;
    const bool logfix = !TR && p.ln_rhs && c00 && comp == 0;
    if (logfix) lnv = *p.ln_rhs * p.ln_scale;
    // IDEL2 (m = 0, k = 0): right-hand side shifted down one row, row 0 <- the LN condition (929-936)
    const bool shift = !TR && HB == 3 && kind == 1 && c00;
    double carry = shift && !comp && fo.has_ln ? fo.ln_in / g.norm0[0] : 0.0;
    // recurrence state: v1, v2, v3 the last values; in the transposed passes the
    // factors of the last rows too (column entries of U, of L)
    double v1 = 0.0, v2 = 0.0, v3 = 0.0, a1 = 0.0, a2 = 0.0, a2p = 0.0, a3 = 0.0, a3p = 0.0, a3q = 0.0;
    for (int c = 0; c < nch; ++c) {
        if (!warp_wait(sh.full + c % SNST, c / SNST, sh)) return -1;
        const double* S = sh.ring + (c % SNST) * (SCH * 64);
        const int lo = c * SCH, rows = min(SCH, size - lo);
        double rb[SCH], f[SCH][HB + 1];
#pragma unroll
        for (int q = 0; q < SCH; ++q) {  // rows past the end read stale values that are not used
            rb[q] = XG && !staged ? (live && q < rows ? sc[(size_t)(lo + q) * st] : 0.0)
                                  : (XG ? (q < rows ? xget(lo + q) : 0.0) : X[(lo + q) * 32]);
            if constexpr (TR) row_u(S + q * WU, f[q]);
            else row_l(S + q * WL, f[q]);
        }
        give_back(sh.empty + c % SNST);
        if (logfix && c == 0) {
            const double cf[3] = {4.0 / 3, -2.0, 2.0 / 3};
#pragma unroll
            for (int q = 0; q < 3; ++q)
                if (q < rows) rb[q] -= lnv * (cf[q] / g.ELL2) / g.norm0[q];
        }
        if (shift) {
            const double last = rb[SCH - 1];
#pragma unroll
            for (int q = SCH - 1; q >= 1; --q) rb[q] = rb[q - 1];
            rb[0] = carry;
            carry = last;
        }
#pragma unroll
        for (int q = 0; q < SCH; ++q) {
            if (q >= rows) break;
            double v = rb[q];
            if constexpr (!TR) {
                if constexpr (HB == 3) v = __fma_rn(-f[q][3], v3, v);
                v = __fma_rn(-f[q][1], v1, __fma_rn(-f[q][2], v2, v));
                xput(lo + q, v);
            } else {
                // w(r) = y(r) - u1(r-1) w(r-1) - u2(r-2) w(r-2) - ..., z(r) = w(r) / U(r, r)
                if constexpr (HB == 3) v = __fma_rn(-a3q, v3, v);
                v = __fma_rn(-a1, v1, __fma_rn(-a2p, v2, v));
                xput(lo + q, __dmul_rn(v, f[q][0]));
                a3q = a3p;
                a3p = a3;
                if constexpr (HB == 3) a3 = f[q][3];
                a2p = a2;
                a2 = f[q][2];
                a1 = f[q][1];
            }
            v3 = v2;
            v2 = v1;
            v1 = v;
        }
    }
    v1 = v2 = v3 = a1 = a2 = a2p = a3 = a3p = a3q = 0.0;
    for (int c = nch; c < 2 * nch; ++c) {
        if (!warp_wait(sh.full + c % SNST, c / SNST, sh)) return -1;
        int lo, rows;
        solve_chunk(c, nch, size, lo, rows);
        const int hi = lo + rows - 1;
        const double* S = sh.ring + (c % SNST) * (SCH * 64);
        double vb[SCH], f[SCH][HB + 1];
#pragma unroll
        for (int q = 0; q < SCH; ++q) {  // rows past the end repeat row lo and are not used
            const int r = max(lo, hi - q);
            vb[q] = xget(r);
            if constexpr (TR) row_l(S + (r - lo) * WL, f[q]);
            else row_u(S + (r - lo) * WU, f[q]);
        }
        give_back(sh.empty + c % SNST);
        if constexpr (!TR) {
#pragma unroll
            for (int q = 0; q < SCH; ++q) vb[q] = __dmul_rn(vb[q], f[q][0]);
        }
#pragma unroll
        for (int q = 0; q < SCH; ++q) {
            if (q >= rows) break;
            double v = vb[q];
            if constexpr (!TR) {
                if constexpr (HB == 3) v = __fma_rn(-f[q][3], v3, v);
                v = __fma_rn(-f[q][1], v1, __fma_rn(-f[q][2], v2, v));
            } else {
                // x(r) = z(r) - L(r+1, r) x(r+1) - L(r+2, r) x(r+2) - ...
                if constexpr (HB == 3) v = __fma_rn(-a3q, v3, v);
                v = __fma_rn(-a1, v1, __fma_rn(-a2p, v2, v));
                a3q = a3p;
                a3p = a3;
                if constexpr (HB == 3) a3 = f[q][3];
                a2p = a2;
                a2 = f[q][2];
                a1 = f[q][1];
            }
            xput(hi - q, v);
            v3 = v2;
            v2 = v1;
            v1 = v;
        }
    }
    if constexpr (TR) {
        if (HB == 3 && nn > 0) {  // row NN - 1 zeroed
            xput(size, 0.0);
            return nn;
        }
        return size;
    } else {
        int rows_out = size;
        if (HB == 3 && kind == 2 && nn > 0) {
            // A(NN) = 0; A(:NN) = XM(:NN) y  (mod_legops.f90:1310-1316)
            xput(nn - 1, 0.0);
            rows_out = nn;
            xm_pass(false);
        }
        if (c00 && size > 0) {
            if (kind == 0) {
                if (!comp) *p.ln_out = __dmul_rn(xget(0), g.norm0[0]);
                xput(0, 0.0);
            } else if (kind == 1 && !comp && p.ln_out) {
                *p.ln_out = fo.has_ln ? __dmul_rn(xget(0), g.norm0[0]) : 0.0;
            }
        }
        if (logfix && p.ln_out) *p.ln_out = lnv;
        if (fo.farfield && m == 0 && size > 0) {
            // a(n=0, m=0, k) -= sum_{n < NRCHOP+pad} AT1(n) a(n, 0, k) / AT1(0); the rows
            // past the system are zero, four partial sums break the chain.  XG has FCH rows'
            // loads in flight (one at a time, the sum was as long as the substitutions)
            constexpr int FCH = XG ? 32 : SCH;
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            for (int r0 = 0; r0 < size; r0 += FCH) {
                double w[FCH], v[FCH];
#pragma unroll
                for (int q = 0; q < FCH; ++q) {
                    const int r = min(r0 + q, size - 1);
                    w[q] = sh.at1[r];
                    v[q] = xget(r);
                }
#pragma unroll
                for (int q = 0; q < FCH; ++q)
                    if (r0 + q < size) s[q & 3] = __fma_rn(w[q], v[q], s[q & 3]);
            }
            const double sum = __dadd_rn(__dadd_rn(s[0], s[1]), __dadd_rn(s[2], s[3]));
            xput(0, __dsub_rn(xget(0), __ddiv_rn(sum, sh.at1[0])));
        }
        return rows_out;
    }
}

template <int HB, bool TR, bool XG>
__device__ __forceinline__ void band_solve(const DevGrid& g, const SolveItem& p, const SolveForm& fo, const double* FL,
                                           const double* FU, int m, int k0, const SolveShared& sh) {
    __shared__ int rows_sh;
    const size_t NK = g.NXCHOPDIM, base = (size_t)m * g.NRCHOPDIM * NK + k0;
    const int nsb = min(16, g.NXCHOPDIM - k0);
    const int nn = max(0, g.NRCHOP + fo.pad - m);
    const int size = max(0, (m == 0 && fo.kind == 2) ? nn - 1 : nn);
    int issued = 0;
    if (threadIdx.x >= 32) {
        issued = solve_producer<HB, TR, XG>(g, p.src + base, nsb, FL, FU, size, nn, sh);
    } else {
        const int rows = solve_consumer<HB, TR, XG>(g, p, fo, m, k0, nsb, size, nn, sh);
        if (threadIdx.x == 0) rows_sh = rows;
    }
    __syncthreads();
    const int rows_out = rows_sh;
    if (rows_out < 0) {  // the consumer stops in any case: without the producer's chunks, or by itself
        if (threadIdx.x == 0 && g.err) *g.err = 1;
        if (threadIdx.x >= 32) solve_drain(issued, sh);
        return;
    }
    const int end = fo.keep_tail ? rows_out : g.NRCHOPDIM, q = threadIdx.x & 15;
    double2* dst = p.dst + base + q;
    if (q >= nsb) return;
#pragma unroll 4
    for (int r = (XG ? rows_out : 0) + (int)(threadIdx.x >> 4); r < end; r += 4)
        dst[(size_t)r * NK] = !XG && r < rows_out ? sh.Xs[r * 16 + q] : make_double2(0.0, 0.0);
}

// doubles of a block's shared memory for columns of `rows` rows (at least SCH, whole chunks)
__host__ __device__ inline size_t solve_doubles(int rows, bool xg) {
    const int r = (rows + SCH - 1) / SCH * SCH;
    return SRING + (xg ? 0 : (size_t)r * 35);
}

template <bool TR, bool XG>
__device__ __forceinline__ void solve_block(const DevGrid& g, const SolveItem& p, const SolveForm& fo, int b) {
    extern __shared__ __align__(128) double sms[];
    __shared__ uint64_t bars[2 * SNST + 1];
    const FactorTable ft(g);
    const int m = b / ft.nkb, kb = b - m * ft.nkb;
    const int R = (max(g.NRCHOP + fo.pad, 0) + 1 + SCH - 1) / SCH * SCH;
    SolveShared sh;
    sh.ring = sms;
    double *at1 = sms + SRING, *xm = at1 + R;
    sh.at1 = XG ? g.at1 : at1;
    sh.xm = XG ? g.xm : xm;
    sh.Xs = (double2*)(xm + 2 * R);
    sh.full = bars;
    sh.empty = bars + SNST;
    sh.whole = bars + 2 * SNST;
    sh.limit = g.wait;
    if (threadIdx.x == 0) {
        for (int q = 0; q < SNST; ++q) {
            bar_init(sh.full + q, 33);
            bar_init(sh.empty + q, 1);
        }
        bar_init(sh.whole, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (b == 0)
            for (int j = 0; j < 2; ++j)
                if (p.ln_dst[j]) *p.ln_dst[j] = *p.ln_src[j];
    }
    if (m == 0 && !XG) {  // the tables of the m = 0 tails
        const int nr = min(R, g.NRCHOPDIM);
        if (fo.farfield)
            for (int r = threadIdx.x; r < nr; r += 64) at1[r] = g.at1[r];
        if (fo.kind == 2)
            for (int r = threadIdx.x; r < 2 * nr; r += 64) xm[r] = g.xm[r];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    const bool wide = m == 0 && (TR ? fo.kind == 2 : fo.kind != 0);
    if (wide) {
        const double* FL = p.F + ft.l7 + (size_t)kb * ft.R * 48;
        const double* FU = p.F + ft.u7 + (size_t)kb * ft.R * 64;
        band_solve<3, TR, XG>(g, p, fo, FL, FU, m, kb * 16, sh);
    } else {
        const size_t blk = (size_t)m * ft.nkb + kb;
        band_solve<2, TR, XG>(g, p, fo, p.F + blk * ft.R * 32, p.F + ft.u5 + blk * ft.R * 48, m, kb * 16, sh);
    }
}

// blockIdx.y: the problem (a step's three viscous solves go in one launch); blocks
// from nblocks on: PROJECT's tail, two axial modes each
template <bool TR, bool XG>
__global__ void __launch_bounds__(64) solve_factored_kernel(DevGrid g, const __grid_constant__ SolveBatch b,
                                                            SolveForm fo, const __grid_constant__ ProjectTail tail,
                                                            int nblocks) {
    if ((int)blockIdx.x >= nblocks) {
        project_tail_warp(g, tail, 2 * (blockIdx.x - nblocks) + (threadIdx.x >> 5), threadIdx.x & 31);
        return;
    }
    solve_block<TR, XG>(g, b.p[blockIdx.y], fo, blockIdx.x);
}

__global__ void __launch_bounds__(64) project_tail_kernel(DevGrid g, const __grid_constant__ ProjectTail tail) {
    project_tail_warp(g, tail, 2 * blockIdx.x + (threadIdx.x >> 5), threadIdx.x & 31);
}

// Grouped form over the instances of an ensemble: a block's problem by binary
// search over `first`.
__global__ void __launch_bounds__(64) grouped_solve_kernel(const GroupSolve* __restrict__ pr,
                                                           const int* __restrict__ first, int np) {
    const int b = blockIdx.x;
    int lo = 0, hi = np - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    const GroupSolve& P = pr[lo];
    solve_block<false, false>(P.g, P.it, SolveForm{P.kind, P.has_ln, P.ln_in, P.pad, P.farfield, 0}, b - P.first);
}

constexpr size_t SOLVE_SMEM_MAX = 220 * 1024;
// g's columns at `pad` with one row to spare (IHELM's row NN at m = 0)
size_t solve_smem(const DevGrid& g, int pad, bool xg) {
    return solve_doubles(std::max(g.NRCHOP + pad, 0) + 1, xg) * sizeof(double);
}

template <class K>
void allow_smem(K kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLVE_SMEM_MAX);
}

template <bool TR>
void launch_solve(const DevGrid& g, const SolveBatch& b, const SolveForm& fo, cudaStream_t s,
                  const ProjectTail* tail = nullptr) {
    static const bool attr = [] {
        allow_smem(solve_factored_kernel<TR, false>);
        allow_smem(solve_factored_kernel<TR, true>);
        return true;
    }();
    (void)attr;
    const int nblocks = FactorTable(g).nkb * g.NTCHOPDIM;
    const dim3 grid(nblocks + (tail ? (g.NXCHOPDIM + 1) / 2 : 0), b.n);
    const ProjectTail tl = tail ? *tail : ProjectTail{};
    const size_t smem = solve_smem(g, fo.pad, false);
    if (smem <= SOLVE_SMEM_MAX) solve_factored_kernel<TR, false><<<grid, 64, smem, s>>>(g, b, fo, tl, nblocks);
    else solve_factored_kernel<TR, true><<<grid, 64, solve_smem(g, fo.pad, true), s>>>(g, b, fo, tl, nblocks);
    count_launch();
}
}  // namespace

void k_solve_factored_batch(const DevGrid& g, const SolveBatch& b, int kind, int has_ln, double ln_in, int pad,
                            int farfield, cudaStream_t s, const ProjectTail* tail) {
    launch_solve<false>(g, b, SolveForm{kind, has_ln, ln_in, pad, farfield, 0}, s, tail);
}

void k_project_tail(const DevGrid& g, const ProjectTail& t, cudaStream_t s) {
    project_tail_kernel<<<(g.NXCHOPDIM + 1) / 2, 64, 0, s>>>(g, t);
    count_launch();
}

void k_solve_factored(const DevGrid& g, const double* F, const double2* src, double2* dst, double* ln_out, int kind,
                      int has_ln, double ln_in, int pad, int farfield, cudaStream_t s, const double* ln_rhs,
                      double ln_scale) {
    SolveBatch b{};
    b.n = 1;
    b.p[0].F = F;
    b.p[0].src = src;
    b.p[0].dst = dst;
    b.p[0].ln_out = ln_out;
    b.p[0].ln_rhs = ln_rhs;
    b.p[0].ln_scale = ln_scale;
    k_solve_factored_batch(g, b, kind, has_ln, ln_in, pad, farfield, s);
}

void k_solve_T(const DevGrid& g, const double* F, double2* y, int kind, int pad, cudaStream_t s) {
    SolveBatch b{};
    b.n = 1;
    b.p[0].F = F;
    b.p[0].src = y;
    b.p[0].dst = y;
    launch_solve<true>(g, b, SolveForm{kind, 0, 0.0, pad, 0, 1}, s);
}

void k_solve_T_batch(const DevGrid& g, const SolveBatch& b, int kind, int pad, cudaStream_t s) {
    launch_solve<true>(g, b, SolveForm{kind, 0, 0.0, pad, 0, 0}, s);
}

int group_solve_blocks(const GroupSolve& p) { return FactorTable(p.g).nkb * p.g.NTCHOPDIM; }
size_t group_solve_smem(const GroupSolve& p) { return solve_smem(p.g, p.pad, false); }

void k_grouped_solve(const GroupSolve* d, const int* first, int np, int total_blocks, size_t smem, cudaStream_t s) {
    static const bool attr = [] {
        allow_smem(grouped_solve_kernel);
        return true;
    }();
    (void)attr;
    grouped_solve_kernel<<<total_blocks, 64, smem, s>>>(d, first, np);
    count_launch();
}

void k_solve_del2(const DevGrid& g, double2* a, double* ln_out, int kind, double alp, int has_ln, double ln_in,
                  const double* b_ln, double* scratch, int pad, cudaStream_t s) {
    int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    solve_kernel<<<(nsys + 63) / 64, 64, 0, s>>>(g, a, ln_out, kind, alp, has_ln, ln_in, b_ln, scratch, pad);
    count_launch();
}

// ---------------------------------------------------------------------------
// IHELMP (mod_legops.f90:1409-1592), the implicit hyperviscosity solve of
// HYPERV (VISC%SW = 2, mod_march.f90:1639-1686): per (m, k) the system
//   H = (DEL2H - k^2)^(P/2) + NU (DEL2H - k^2) - ALP
// of half-bandwidth P on the leading NN = NRCHOP + pad - m rows.  H's rows are
// formed from the powers D^q of the DEL2H band (table dq, built on the host
// with BANBANMUL's summation order), combined binomially as the reference
// writes them out for each P (D^(P/2) - C(P/2,1) k^2 D^(P/2-1) + ... ), then
// eliminated without pivoting, one thread per (m, k), the U rows in scratch
// [row][P+1][system], the right-hand side in place.  The (m, k) = (0, 0)
// thread first moves the log term's contribution to the right-hand side:
// rows -= AL + NU AL2, AL2 the DEL2 image of LN (-log(1-x)) and AL = D^(P/2-1) AL2.
// dq layout: [m][q = 1..HP][row < rows][4q + 1], q's block at rows (q - 1)(2q + 1)
// within the m block of rows HP (2 HP + 3) doubles.
template <int HP>
__global__ void ihelmp_kernel(DevGrid g, const double* dq, int rows, double2* A, const double* ln, double alp,
                              double nu, double* scratch, int pad) {
    constexpr int P = 2 * HP, W = 2 * P + 1;
    const int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsys) return;
    const int k = t % g.NXCHOPDIM;
    const int m = t / g.NXCHOPDIM;
    int nn = g.NRCHOP + pad - m;
    if (nn > rows) nn = rows;
    if (nn <= 0) return;
    const double K2 = g.ak[k] * g.ak[k];
    const size_t mstride = (size_t)rows * HP * (2 * HP + 3);  // rows * sum_{q <= HP} (4q + 1)
    const double* dm = dq + (size_t)m * mstride;
    // q's block starts after rows * sum_{q' < q} (4q' + 1) = rows (q - 1)(2q + 1)
    auto dq_row = [&](int q, int r) { return dm + (size_t)rows * (q - 1) * (2 * q + 1) + (size_t)r * (4 * q + 1); };
    double2* col = A + (size_t)m * g.NRCHOPDIM * g.NXCHOPDIM + k;
    const size_t st = g.NXCHOPDIM;
    if (m == 0 && k == 0) {
        // log term (1444-1466): A%LN was set to -B%LN/ALP by the caller
        const int nr = g.NRCHOP + pad;
        const double L = *ln;
        double al2[P + 3], al[P + 3], y[P + 3];
        for (int i = 0; i < P + 3; ++i) al2[i] = 0.0;
        al2[0] = L * (4.0 / 3 / g.ELL2) / g.norm0[0];
        al2[1] = L * (-2 / g.norm0[1] / g.ELL2);
        al2[2] = L * (+2.0 / 3 / g.norm0[2] / g.ELL2);
        for (int i = 0; i < P + 3; ++i) al[i] = al2[i];
        const double* d2 = g.del2h;  // m = 0 rows, [row][5]
        for (int rep = 1; rep < HP; ++rep) {  // BANMUL(DEL2H, 3, AL), band index ascending
            for (int r = 0; r < P + 3; ++r) {
                double v = 0.0;
                for (int e = 0; e < 5; ++e) {
                    const int c = r + e - 2;
                    if (r < nr && c >= 0 && c < nr && c < P + 3) v += d2[(size_t)r * 5 + e] * al[c];
                }
                y[r] = v;
            }
            for (int r = 0; r < P + 3; ++r) al[r] = y[r];
        }
        for (int r = 0; r < P + 3 && r < nr; ++r) {
            double2 v = col[(size_t)r * st];
            v.x -= al[r] + nu * al2[r];
            col[(size_t)r * st] = v;
        }
    }
    // forward elimination, left-looking per row (the pivot rows come from scratch)
    for (int r = 0; r < nn; ++r) {
        double w[W];
        const double* top = dq_row(HP, r);
#pragma unroll
        for (int e = 0; e < W; ++e) w[e] = top[e];
        double c = 1.0;
#pragma unroll
        for (int j = 1; j <= HP; ++j) {
            c *= -K2;
            // binomial coefficient C(HP, j)
            double bin = 1.0;
            for (int q = 1; q <= j; ++q) bin = bin * (HP - q + 1) / q;
            const int q = HP - j;
            if (q == 0) {
                w[P] += c;
            } else {
                const double* dr = dq_row(q, r);
                const double f = bin * c;
                for (int e = 0; e <= 4 * q; ++e) w[P - 2 * q + e] += f * dr[e];
            }
        }
        {
            const double* d1 = dq_row(1, r);
            for (int e = 0; e < 5; ++e) w[P - 2 + e] += nu * (e == 2 ? d1[e] - K2 : d1[e]);
        }
        w[P] -= alp;
        double2 rhs = col[(size_t)r * st];
        for (int d = P; d >= 1; --d) {
            if (r - d < 0) continue;
            const double* u = scratch + (size_t)(r - d) * (P + 1) * nsys + t;
            const double f = w[P - d] / u[0];
            w[P - d] = 0.0;
            for (int j = 1; j <= P; ++j) {
                const int qq = P - d + j;
                if (qq < W) w[qq] -= f * u[(size_t)j * nsys];
            }
            const double2 pr = col[(size_t)(r - d) * st];
            rhs.x -= f * pr.x;
            rhs.y -= f * pr.y;
        }
        double* ur = scratch + (size_t)r * (P + 1) * nsys + t;
        for (int j = 0; j <= P; ++j) ur[(size_t)j * nsys] = w[P + j];
        col[(size_t)r * st] = rhs;
    }
    // back substitution
    for (int r = nn - 1; r >= 0; --r) {
        const double* ur = scratch + (size_t)r * (P + 1) * nsys + t;
        double2 v = col[(size_t)r * st];
        for (int j = 1; j <= P && r + j < nn; ++j) {
            const double u = ur[(size_t)j * nsys];
            const double2 x = col[(size_t)(r + j) * st];
            v.x -= u * x.x;
            v.y -= u * x.y;
        }
        v.x /= ur[0];
        v.y /= ur[0];
        col[(size_t)r * st] = v;
    }
}

size_t ihelmp_scratch_doubles(const DevGrid& g, int P) {
    return (size_t)g.NRCHOPDIM * (P + 1) * g.NTCHOPDIM * g.NXCHOPDIM;
}

void k_ihelmp(const DevGrid& g, int P, const double* dq, int rows, double2* a, const double* ln, double alp,
              double nu, double* scratch, int pad, cudaStream_t s) {
    const int nsys = g.NTCHOPDIM * g.NXCHOPDIM;
    const int bs = 128, nb = (nsys + bs - 1) / bs;
    switch (P) {
        case 4: ihelmp_kernel<2><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
        case 6: ihelmp_kernel<3><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
        case 8: ihelmp_kernel<4><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
        case 10: ihelmp_kernel<5><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
        case 12: ihelmp_kernel<6><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
        default: ihelmp_kernel<7><<<nb, bs, 0, s>>>(g, dq, rows, a, ln, alp, nu, scratch, pad); break;
    }
    count_launch();
}

}  // namespace mlegs
