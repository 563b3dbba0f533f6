// fp64.cu -- the FP64 parity engine (fp64.h): the reference's -DDOUBLE timestep on the GPU.
//
// State lives in tag order as wrapped FP64 positions, velocities, forces and image counters.
// Each step: the initial half kick and drift with wrapping (src/fix/fix_nve.cu:42-86), a
// cell grid of fixed-capacity cells (indices appended by atomics, then each cell's records
// written in index order so the summation order is fixed), the mDPD density pass
// (src/force/pair_mdpd.cu:253-297), the force pass, the final half kick
// (src/fix/fix_nve.cu:131-149) and on logged steps a fixed-order reduction of the thermo sums
// (src/compute/thermo.cu:240-246,301-303,422-434,506-517).  The force pass gives one warp all
// pairs of a cell's atoms from both sides (the 27 cells' candidates staged once, the pairs
// inside the cutoff evaluated 32 at a time), their bonds and angles, summed by fixed trees, so
// no atomics touch the forces and runs repeat bit for bit.
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "dpd_common.h"
#include "fp64.h"
#include "launch_rules.h"
#include "saru.cuh"

namespace dpd {

namespace {

enum { F64_NONFINITE = 1, F64_FENE = 2, F64_CELL_OVERFLOW = 4, F64_FAR = 8 };
enum { NQ = 9, NSUM = 19, RED_BLOCKS = 256 };
// pair table per type pair: A, B, gamma, rc, rd, sigma = sqrt(gamma) sqrt(2 kT)/sqrt(dt),
// 1/rc, 1/rd, rc^2
enum { NC = 9 };

struct F64Args {
    int n, ntypes, style, bond_style, angle_style, cap;
    int nc[3];
    uint32_t seed, integ_mask;
    double lo[3], L[3], w[3], dt, maxrc2;
    const double *coeff, *mass, *bondc, *anglec;
    double *x, *v, *f, *rho, *q;
    double *xn, *vn;  // the next step's positions and velocities (fused step)
    int *img, *type, *cnt, *status;
    int* cnt_next;    // cell counts of the next binning, cleared by this step's sort
    int *owner, *owner_prev;  // sparse boxes: an atom's cell where it came first, else -1; the binning before
    int* craw;      // atom indices appended to each cell, cap per cell
    double4* crec;  // cell records in index order: position and atom index (rec_index)
    int* ccode;  // each atom's cell as cx | cy << 10 | cz << 20, written by the binning
    const int *bstart, *astart;
    const int2* bent;
    const int4* aent;
};

// minimum image, src/force/neigh_list.cu:377-379: d -= L*((d >= L/2) - (d < -L/2))
__device__ __forceinline__ double min_image(double d, double L)
{
    const double h = 0.5 * L;
    return d - (d >= h ? L : (d < -h ? -L : 0.0));
}

// the atom index of a cell record, kept as the bits of its fourth word
__device__ __forceinline__ double rec_word(int i) { return __longlong_as_double((long long)i); }
__device__ __forceinline__ int rec_index(const double4& r) { return (int)__double_as_longlong(r.w); }

// triangular type-pair index, src/force/pair_dpd.cu:134 (types 1-based, result 0-based)
__device__ __forceinline__ int tri(int ti, int tj, int nt)
{
    const int a = min(ti, tj), b = max(ti, tj);
    return ((a - 1) * nt - (a - 1) * (a - 2) / 2 + b - a + 1) - 1;
}

// Kernels launched with programmatic dependent launch wait here until their predecessor's
// memory is visible; without a programmatic predecessor the wait returns at once.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ int cell_of(const F64Args& a, const double* p, int c[3])
{
#pragma unroll
    for (int d = 0; d < 3; d++) {
        int k = (int)floor((p[d] - a.lo[d]) / a.w[d]);
        c[d] = min(max(k, 0), a.nc[d] - 1);
    }
    return (c[0] * a.nc[1] + c[1]) * a.nc[2] + c[2];
}

// an atom into its cell (appended in the order the atomics draw)
__device__ __forceinline__ void bin_atom(const F64Args& a, int i, const double* x, int* cnt)
{
    int c[3];
    const int cell = cell_of(a, x, c);
    a.ccode[i] = c[0] | (c[1] << 10) | (c[2] << 20);
    const int k = atomicAdd(cnt + cell, 1);
    if (k < a.cap) a.craw[(size_t)cell * a.cap + k] = i;
    else atomicOr(a.status, F64_CELL_OVERFLOW);
}

__global__ void k64_bin(F64Args a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.n) bin_atom(a, i, a.x + 3 * i, a.cnt);
}

// each cell's records in atom-index order, so the pair sums run in a fixed order: 8 lanes per
// cell rank its indices (a record's place is the number of smaller indices) and gather the
// records; the counts that the next binning starts from are cleared
__global__ void __launch_bounds__(256) k64_sort_cells(F64Args a, int ncell)
{
    dep_wait();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = g >> 3;
    if (c >= ncell) return;
    const int* raw = a.craw + (size_t)c * a.cap;
    const int m = min(a.cnt[c], a.cap);
    if ((g & 7) == 0) a.cnt_next[c] = 0;
    for (int k = g & 7; k < m; k += 8) {
        const int i = raw[k];
        int place = 0;
        for (int q = 0; q < m; q++) place += raw[q] < i;
        const size_t to = (size_t)c * a.cap + place;
        a.crec[to] = make_double4(a.x[3 * i], a.x[3 * i + 1], a.x[3 * i + 2], rec_word(i));
    }
}

// Sparse boxes: the records appended as the atomics draw; the atom that comes first in a cell owns it
__global__ void k64_bin_owned(F64Args a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    int c[3];
    const double x[3] = {a.x[3 * i], a.x[3 * i + 1], a.x[3 * i + 2]};
    const int cell = cell_of(a, x, c);
    a.ccode[i] = c[0] | (c[1] << 10) | (c[2] << 20);
    const int k = atomicAdd(a.cnt + cell, 1);
    a.owner[i] = k == 0 ? cell : -1;
    if (k < a.cap) a.crec[(size_t)cell * a.cap + k] = make_double4(x[0], x[1], x[2], rec_word(i));
    else atomicOr(a.status, F64_CELL_OVERFLOW);
}

// and sorted, a thread per owner (most cells have one record); the counts of the cells that were
// owned in the binning before are cleared, so that no pass goes over the empty cells
__global__ void k64_sort_owned(F64Args a)
{
    dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int prev = a.owner_prev[i], c = a.owner[i];
    if (prev >= 0) a.cnt_next[prev] = 0;
    if (c < 0) return;
    double4* l = a.crec + (size_t)c * a.cap;
    const int m = min(a.cnt[c], a.cap);
    for (int p = 1; p < m; p++) {
        const double4 v = l[p];
        int q = p - 1;
        while (q >= 0 && rec_index(l[q]) > rec_index(v)) {
            l[q + 1] = l[q];
            q--;
        }
        l[q + 1] = v;
    }
}

// the c-th of the 27 cells around atom i (c = 9 (ox+1) + 3 (oy+1) + (oz+1); nc >= 3 per
// dimension, so no cell is visited twice); calls fn(j, dx, dy, dz, r2) for every other
// atom j there with r2 <= maxrc2, in index order
template <class F>
__device__ __forceinline__ void for_cell(const F64Args& a, int i, int c, F&& fn)
{
    const double xi = a.x[3 * i], yi = a.x[3 * i + 1], zi = a.x[3 * i + 2];
    const int code = a.ccode[i];
    int cx = (code & 1023) + c / 9 - 1, cy = ((code >> 10) & 1023) + (c / 3) % 3 - 1, cz = (code >> 20) + c % 3 - 1;
    cx += cx < 0 ? a.nc[0] : 0; cx -= cx >= a.nc[0] ? a.nc[0] : 0;
    cy += cy < 0 ? a.nc[1] : 0; cy -= cy >= a.nc[1] ? a.nc[1] : 0;
    cz += cz < 0 ? a.nc[2] : 0; cz -= cz >= a.nc[2] ? a.nc[2] : 0;
    const int cell = (cx * a.nc[1] + cy) * a.nc[2] + cz;
    const double4* l = a.crec + (size_t)cell * a.cap;
    const int m = min(a.cnt[cell], a.cap);
    for (int p = 0; p < m; p++) {
        const double4 rj = l[p];
        const int j = rec_index(rj);
        if (j == i) continue;
        const double dx = min_image(xi - rj.x, a.L[0]);
        const double dy = min_image(yi - rj.y, a.L[1]);
        const double dz = min_image(zi - rj.z, a.L[2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 <= a.maxrc2) fn(j, dx, dy, dz, r2);
    }
}

// sum over the warp by a fixed butterfly: the same order on every run
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// mDPD local density, src/force/pair_mdpd.cu:253-297: rho_i = sum_{j != i}
// 15/(2 pi rd^3) max(0, 1 - r/rd)^2 (pairs within the largest cutoff).  One warp per
// atom, lane c takes the c-th of the 27 cells.
__global__ void __launch_bounds__(256) k64_density(F64Args a)
{
    dep_wait();
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= a.n) return;  // warp-uniform
    const int ti = a.type[i];
    double rho = 0.0;
    if (lane < 27)
        for_cell(a, i, lane, [&](int j, double, double, double, double r2) {
            const double* c = a.coeff + NC * tri(ti, a.type[j], a.ntypes);
            const double rd = c[4];
            double wd = 1.0 - sqrt(r2) * c[7];
            if (wd < 0.0) wd = 0.0;
            rho += 15.0 / 2.0 / 3.14159265358979323846 / (rd * rd * rd) * wd * wd;
        });
    rho = warp_sum(rho);
    if (lane == 0) a.rho[i] = rho;
}

__device__ __forceinline__ bool integrated(const F64Args& a, int t)
{
    return !a.integ_mask || ((a.integ_mask >> (t - 1)) & 1u);
}

// a drifted coordinate with the reference's wrap (a while loop moving whole box lengths and
// counting images); a non-finite coordinate, or one more than 4 box lengths away after a
// step, is an error
__device__ __forceinline__ double wrap_coord(const F64Args& a, double p, int d, int* img)
{
    const double hi = a.lo[d] + a.L[d];
    if (!isfinite(p)) {
        atomicOr(a.status, F64_NONFINITE);
        p = a.lo[d];
    }
    int guard = 0;
    while ((p >= hi || p < a.lo[d]) && guard < 4) {
        const int k = (p >= hi) - (p < a.lo[d]);
        p -= a.L[d] * k;
        *img += k;
        guard++;
    }
    if (p >= hi || p < a.lo[d]) {
        atomicOr(a.status, F64_FAR);
        p = a.lo[d];
    }
    return p;
}

// Forces, one warp per cell.  The records of the 27 cells around it (src/force/pair_dpd.cu:
// 292-403, pair_mdpd.cu:399-521) are staged in shared memory once, cell by cell in a fixed
// order and each cell's records in index order; the cell's atoms are then taken one after the
// other, each against the staged records 32 at a time, and the pairs inside the largest cutoff
// are queued in ballot order.  Whenever 32 are queued every lane evaluates one (the Saru random
// force, the FP64 force) and a segmented tree over the lanes sums the pairs of each atom, so
// the queue is shared by the cell's atoms and the sums repeat bit for bit.  Four lanes per atom
// share out its bonds (src/force/bond_harmonic.cu:208-268; FENE + WCA as the FP32 engine) and
// harmonic angles (src/force/angle_harmonic.cu:187-270).  STEP: the warp holds its atoms' whole
// forces, so it also takes them through the final half kick, the next step's initial half kick
// and drift, and appends them to their next cells (positions and velocities into the other
// buffers, which no warp of this launch reads); a step without thermo is then this kernel and
// the sort in place of six (3000 atoms 34 -> 16 us, 24000 51 -> 34, 192000 206 -> 192, 648000
// 658 either way).  On logged steps the atom's share of
// the energies and of the virial: half of each pair and bond, a third of each angle, as the
// reference splits them.
// Issue and latency bound it (54% of the issue slots, 20 to 28 warps per SM by registers).
// With a warp per atom every atom found its candidates' cells anew and its 12.6 pairs ran on
// 32 lanes (1048 warp instructions an atom); a whole step of the 192k melt went from 279 to
// 206 us, of the 648k melt from 924 to 658, of 24k from 63 to 51.  7 blocks per SM; 8 and 10
// spill (211 and 227 us at 192k).  Velocities beside the records instead of by atom index: no
// gain (231 against 228 us) for twice the cell memory.
#define F64_Q 64      // queued pairs (power of two, >= 63)
#define F64_TILE 128  // staged records (27 cells of about 3 atoms, more in several rounds)
#define F64_HOME 8    // atoms of the cell taken per round
#define F64_WARPS 4   // warps per block

template <bool LOG>
struct F64Warp {
    static constexpr int NV = LOG ? 10 : 3;  // fx fy fz [pe, virial]
    double4 rec[F64_TILE];                   // staged: position (the image next to the cell), index
    double4 hx[F64_HOME], hv[F64_HOME];      // the round's atoms: position, index; velocity, type
    double acc[F64_HOME][NV];
    double rho[F64_HOME];
    unsigned short q[F64_Q];                 // queued: staged record * F64_HOME + home atom
};

// one pair inside the largest cutoff: the force on i and the pair energy; false outside its own cutoff
__device__ __forceinline__ bool f64_pair(const F64Args& a, uint32_t step, int i, int j, int ti, double dx, double dy,
                                         double dz, double r2, double dvx, double dvy, double dvz, const double& rho_i,
                                         double& gx, double& gy, double& gz, double& e2)
{
    const double* c = a.coeff + NC * tri(ti, a.type[j], a.ntypes);
    // 1/r by rsqrt and r/rc as r * (1/rc): within an ulp of the divisions
    const double rinv = rsqrt(r2);
    const double r = r2 * rinv;
    if (!(r2 <= c[8]) || r < 1.0e-10) return false;
    const double A = c[0], B = c[1], gamma = c[2], rc = c[3], rd = c[4], sigma = c[5];
    const double dot = dx * dvx + dy * dvy + dz * dvz;
    const double wc = 1.0 - r * c[6];
    const uint32_t t1 = (uint32_t)min(i, j) + 1u, t2 = (uint32_t)max(i, j) + 1u;
    const double theta = saru_theta_f64(t1, t2, a.seed, step);
    double fpair;
    if (a.style == 0) {
        fpair = A * wc - gamma * wc * wc * dot * rinv + sigma * wc * theta;
        e2 = 0.5 * A * rc * wc * wc;
    } else {
        double wd = 1.0 - r * c[7];
        if (wd < 0.0) wd = 0.0;
        const double rs = rho_i + a.rho[j];
        fpair = A * wc + B * rs * wd - gamma * wc * wc * dot * rinv + sigma * wc * theta;
        e2 = 0.5 * A * rc * wc * wc + 0.25 * B * rd * rs * wd * wd;
    }
    fpair *= rinv;
    gx = dx * fpair;
    gy = dy * fpair;
    gz = dz * fpair;
    return true;
}

// the first cnt queued pairs from `head`, one per lane, added to their atoms' sums
template <bool LOG>
__device__ __forceinline__ void f64_pairs(const F64Args& a, uint32_t step, F64Warp<LOG>& w, uint32_t head, int cnt,
                                          int lane)
{
    constexpr int NV = F64Warp<LOG>::NV;
    double val[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) val[k] = 0.0;
    int h = F64_HOME + lane;  // lanes without a pair: segments of their own
    if (lane < cnt) {
        const unsigned q = w.q[(head + lane) & (F64_Q - 1)];
        h = (int)(q & (F64_HOME - 1));
        const double4 xj = w.rec[q / F64_HOME], xi = w.hx[h], vi = w.hv[h];
        const int i = rec_index(xi), j = rec_index(xj);
        const double dvx = vi.x - a.v[3 * j], dvy = vi.y - a.v[3 * j + 1], dvz = vi.z - a.v[3 * j + 2];
        const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        const double r2 = dx * dx + dy * dy + dz * dz;
        double gx, gy, gz, e2;
        if (f64_pair(a, step, i, j, rec_index(vi), dx, dy, dz, r2, dvx, dvy, dvz, w.rho[h], gx, gy, gz, e2)) {
            val[0] = gx;
            val[1] = gy;
            val[2] = gz;
            if (LOG) {
                val[NV - 7] = 0.5 * e2;
                val[NV - 6] = 0.5 * dx * gx; val[NV - 5] = 0.5 * dx * gy; val[NV - 4] = 0.5 * dx * gz;
                val[NV - 3] = 0.5 * dy * gy; val[NV - 2] = 0.5 * dy * gz; val[NV - 1] = 0.5 * dz * gz;
            }
        }
    }
    // the pairs of an atom are on consecutive lanes: a fixed tree within each segment
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const bool same = __shfl_down_sync(0xffffffffu, h, o) == h && lane + o < 32;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const double t = __shfl_down_sync(0xffffffffu, val[k], o);
            if (same) val[k] += t;
        }
    }
    const int before = __shfl_up_sync(0xffffffffu, h, 1);
    if (h < F64_HOME && (lane == 0 || before != h))
#pragma unroll
        for (int k = 0; k < NV; k++) w.acc[h][k] += val[k];
    __syncwarp();
}

// atom i's bonds and angles, every `lanes`-th from the sub-th, added to the lane's sums
template <bool LOG>
__device__ __forceinline__ void f64_bonded(const F64Args& a, int i, int sub, int lanes, double& fx, double& fy,
                                           double& fz, double& bpe, double& ape, double (&vir)[6])
{
    for (int b = a.bstart[i] + sub; b < a.bstart[i + 1]; b += lanes) {
        const int2 e2 = a.bent[b];
        const int j = e2.x;
        const double dx = min_image(a.x[3 * i] - a.x[3 * j], a.L[0]);
        const double dy = min_image(a.x[3 * i + 1] - a.x[3 * j + 1], a.L[1]);
        const double dz = min_image(a.x[3 * i + 2] - a.x[3 * j + 2], a.L[2]);
        const double r2 = dx * dx + dy * dy + dz * dz;
        const double r = sqrt(r2);
        const double* bc = a.bondc + 4 * (e2.y - 1);
        double fbond = 0.0, e = 0.0;
        if (a.bond_style == 1) {
            fbond = r > 0.0 ? -2.0 * bc[0] * (r - bc[1]) / r : 0.0;
            e = bc[0] * (r - bc[1]) * (r - bc[1]);
        } else if (a.bond_style == 2) {
            const double K = bc[0], R0 = bc[1], eps = bc[2], sg = bc[3];
            double rr = r2 / (R0 * R0);
            if (rr >= 1.0) {
                atomicOr(a.status, F64_FENE);
                rr = 0.999;
            }
            fbond = -K / (1.0 - rr);
            e = -0.5 * K * R0 * R0 * log(1.0 - rr);
            if (eps > 0.0 && r2 < 1.2599210498948731647672106 * sg * sg) {  // 2^(1/3) s^2
                const double sr2 = sg * sg / r2, sr6 = sr2 * sr2 * sr2;
                fbond += 48.0 * eps * sr6 * (sr6 - 0.5) / r2;
                e += 4.0 * eps * sr6 * (sr6 - 1.0) + eps;
            }
        }
        const double gx = dx * fbond, gy = dy * fbond, gz = dz * fbond;
        fx += gx;
        fy += gy;
        fz += gz;
        if (LOG) {
            bpe += 0.5 * e;
            vir[0] += 0.5 * dx * gx; vir[1] += 0.5 * dx * gy; vir[2] += 0.5 * dx * gz;
            vir[3] += 0.5 * dy * gy; vir[4] += 0.5 * dy * gz; vir[5] += 0.5 * dz * gz;
        }
    }
    for (int t = a.astart[i] + sub; t < a.astart[i + 1]; t += lanes) {
        const int4 an = a.aent[t];
        double d1[3], d2[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            d1[c] = min_image(a.x[3 * an.x + c] - a.x[3 * an.y + c], a.L[c]);
            d2[c] = min_image(a.x[3 * an.z + c] - a.x[3 * an.y + c], a.L[c]);
        }
        const double rsq1 = d1[0] * d1[0] + d1[1] * d1[1] + d1[2] * d1[2];
        const double rsq2 = d2[0] * d2[0] + d2[1] * d2[1] + d2[2] * d2[2];
        const double r1 = sqrt(rsq1), r2 = sqrt(rsq2);
        double c = (d1[0] * d2[0] + d1[1] * d2[1] + d1[2] * d2[2]) / (r1 * r2);
        c = fmin(fmax(c, -1.0), 1.0);
        double s = sqrt(1.0 - c * c);
        if (s < 0.001) s = 0.001;
        const double kk = a.anglec[2 * (an.w - 1)];
        const double theta0 = a.anglec[2 * (an.w - 1) + 1] * (3.14159265358979323846 / 180.0);
        const double dth = acos(c) - theta0;
        const double aa = -2.0 * kk * dth / s;
        const double a11 = aa * c / rsq1, a12 = -aa / (r1 * r2), a22 = aa * c / rsq2;
        double fi[3], fk[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            fi[q] = a11 * d1[q] + a12 * d2[q];
            fk[q] = a22 * d2[q] + a12 * d1[q];
        }
        if (i == an.x) {
            fx += fi[0]; fy += fi[1]; fz += fi[2];
        } else if (i == an.z) {
            fx += fk[0]; fy += fk[1]; fz += fk[2];
        } else {
            fx -= fi[0] + fk[0]; fy -= fi[1] + fk[1]; fz -= fi[2] + fk[2];
        }
        if (LOG) {
            const double third = 1.0 / 3.0;
            ape += third * kk * dth * dth;
            vir[0] += third * (d1[0] * fi[0] + d2[0] * fk[0]);
            vir[1] += third * (d1[0] * fi[1] + d2[0] * fk[1]);
            vir[2] += third * (d1[0] * fi[2] + d2[0] * fk[2]);
            vir[3] += third * (d1[1] * fi[1] + d2[1] * fk[1]);
            vir[4] += third * (d1[1] * fi[2] + d2[1] * fk[2]);
            vir[5] += third * (d1[2] * fi[2] + d2[2] * fk[2]);
        }
    }
}

template <bool LOG, bool STEP>
__global__ void __launch_bounds__(F64_WARPS * 32, LOG ? 4 : 7) k64_force(F64Args a, uint32_t step, int ncell)
{
    dep_wait();
    extern __shared__ double4 f64_smem[];
    constexpr int NV = F64Warp<LOG>::NV;
    F64Warp<LOG>& w = reinterpret_cast<F64Warp<LOG>*>(f64_smem)[threadIdx.x >> 5];
    const int home = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (home >= ncell) return;  // warp-uniform
    const int m0 = min(a.cnt[home], a.cap);
    if (m0 == 0) return;
    // lane c < 27: the c-th cell around the home cell (c = 9 (ox+1) + 3 (oy+1) + (oz+1); nc >= 3
    // per dimension, so no cell is visited twice), its record count, and the box lengths that
    // bring its atoms next to the home cell (-1, 0, 1 per dimension).  A pair inside the cutoff
    // lies in neighbouring cells, so that image is the nearest one.
    int cell = 0, m = 0, img = 0;
    if (lane < 27) {
        int cx = home / (a.nc[1] * a.nc[2]) + lane / 9 - 1, cy = (home / a.nc[2]) % a.nc[1] + (lane / 3) % 3 - 1,
            cz = home % a.nc[2] + lane % 3 - 1;
        const int wx = (cx >= a.nc[0]) - (cx < 0), wy = (cy >= a.nc[1]) - (cy < 0), wz = (cz >= a.nc[2]) - (cz < 0);
        cell = ((cx - wx * a.nc[0]) * a.nc[1] + cy - wy * a.nc[1]) * a.nc[2] + cz - wz * a.nc[2];
        img = (wx + 1) | (wy + 1) << 2 | (wz + 1) << 4;
        m = min(a.cnt[cell], a.cap);
    }
    int incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int excl = incl - m;
    const int M = __shfl_sync(0xffffffffu, incl, 31);
    const unsigned lt = (1u << lane) - 1u;
    for (int h0 = 0; h0 < m0; h0 += F64_HOME) {
        const int nh = min(F64_HOME, m0 - h0);
        if (lane < nh) {
            const double4 x = a.crec[(size_t)home * a.cap + h0 + lane];
            w.hx[lane] = x;
            const int i = rec_index(x);
            w.hv[lane] = make_double4(a.v[3 * i], a.v[3 * i + 1], a.v[3 * i + 2], rec_word(a.type[i]));
            if (a.style == 1) w.rho[lane] = a.rho[i];
#pragma unroll
            for (int k = 0; k < NV; k++) w.acc[lane][k] = 0.0;
        }
        uint32_t head = 0, tail = 0;
        for (int tb = 0; tb < M; tb += F64_TILE) {
            const int nt = min(F64_TILE, M - tb);
            if (h0 == 0 || M > F64_TILE) {
                for (int q = lane; q < nt + lane; q += 32) {  // uniform trip count (shuffles)
                    const int t = tb + q;
                    // the candidate's cell: the last of the 27 whose first record is at or
                    // before t (an empty cell shares its start with the next one, which then wins)
                    int c = 0;
#pragma unroll
                    for (int stp = 16; stp >= 1; stp >>= 1) {
                        const int probe = min(c + stp, 26);
                        const int pstart = __shfl_sync(0xffffffffu, excl, probe);
                        if (c + stp <= 26 && pstart <= t) c += stp;
                    }
                    const int cc = __shfl_sync(0xffffffffu, cell, c);
                    const int c0 = __shfl_sync(0xffffffffu, excl, c);
                    const int im = __shfl_sync(0xffffffffu, img, c);
                    if (q < nt) {
                        // the box length is added to the neighbour before the difference is
                        // taken, so across the boundary the two sides of a pair are negatives of
                        // each other to the last bit of the coordinate, not exactly; the error
                        // against the exact difference is the same
                        double4 rj = a.crec[(size_t)cc * a.cap + (t - c0)];
                        rj.x += (im & 3) == 1 ? 0.0 : ((im & 3) ? a.L[0] : -a.L[0]);
                        rj.y += ((im >> 2) & 3) == 1 ? 0.0 : (((im >> 2) & 3) ? a.L[1] : -a.L[1]);
                        rj.z += (im >> 4) == 1 ? 0.0 : ((im >> 4) ? a.L[2] : -a.L[2]);
                        w.rec[q] = rj;
                    }
                }
            }
            __syncwarp();
            for (int h = 0; h < nh; h++) {
                const double4 xi = w.hx[h];
                const int i0 = rec_index(xi);
                for (int q = lane; q < nt + lane; q += 32) {
                    bool hit = false;
                    if (q < nt) {
                        const double4 rj = w.rec[q];
                        const double dx = xi.x - rj.x, dy = xi.y - rj.y, dz = xi.z - rj.z;
                        hit = rec_index(rj) != i0 && dx * dx + dy * dy + dz * dz <= a.maxrc2;
                    }
                    const unsigned bm = __ballot_sync(0xffffffffu, hit);
                    if (hit) w.q[(tail + __popc(bm & lt)) & (F64_Q - 1)] = (unsigned short)(q * F64_HOME + h);
                    tail += __popc(bm);
                    if (tail - head >= 32u) {
                        __syncwarp();
                        f64_pairs<LOG>(a, step, w, head, 32, lane);
                        head += 32;
                    }
                }
            }
            // the rest of the queue: its atoms come again with the next staged records, and a
            // chunk's pairs of one atom have to be neighbours
            __syncwarp();
            if (tail != head) f64_pairs<LOG>(a, step, w, head, (int)(tail - head), lane);
            head = tail;
        }
        // bonds and angles: lanes 4 h .. 4 h + 3 for the round's atom h
        static_assert(F64_HOME * 4 == 32, "four lanes per atom of a round");
        const int h = lane >> 2, sub = lane & 3;
        double fx = 0.0, fy = 0.0, fz = 0.0, bpe = 0.0, ape = 0.0;
        double vir[6] = {0, 0, 0, 0, 0, 0};
        const int i = h < nh ? rec_index(w.hx[h]) : 0;
        if (h < nh) f64_bonded<LOG>(a, i, sub, 4, fx, fy, fz, bpe, ape, vir);
        auto sum4 = [](double v) {
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            return v;
        };
        fx = sum4(fx);
        fy = sum4(fy);
        fz = sum4(fz);
        if (LOG) {
            bpe = sum4(bpe);
            ape = sum4(ape);
#pragma unroll
            for (int k = 0; k < 6; k++) vir[k] = sum4(vir[k]);
        }
        double p = 0.0;
        if (h < nh && sub < 3) {  // a lane per component
            const double f = w.acc[h][sub] + (sub == 0 ? fx : (sub == 1 ? fy : fz));
            a.f[3 * i + sub] = f;
            if (STEP) {
                const double4 xi = w.hx[h], vi = w.hv[h];
                double v = sub == 0 ? vi.x : (sub == 1 ? vi.y : vi.z);
                p = sub == 0 ? xi.x : (sub == 1 ? xi.y : xi.z);
                const int t = rec_index(vi);
                if (integrated(a, t)) {
                    const double dtm = 0.5 * a.dt / a.mass[t - 1];
                    v += dtm * f;
                    v += dtm * f;
                    p = wrap_coord(a, p + a.dt * v, sub, a.img + 3 * i + sub);
                }
                a.vn[3 * i + sub] = v;
                a.xn[3 * i + sub] = p;
            }
        }
        if (STEP) {
            const double py = __shfl_sync(0xffffffffu, p, (lane & ~3) + 1), pz = __shfl_sync(0xffffffffu, p, (lane & ~3) + 2);
            if (h < nh && sub == 0) {
                const double at[3] = {p, py, pz};
                bin_atom(a, i, at, a.cnt_next);
            }
        }
        if (h < nh && sub == 0) {
            if (LOG) {
                double* q = a.q + (size_t)NQ * i;
                q[0] = w.acc[h][NV - 7];
                q[1] = bpe;
                q[2] = ape;
#pragma unroll
                for (int k = 0; k < 6; k++) q[3 + k] = w.acc[h][NV - 6 + k] + vir[k];
            }
        }
        __syncwarp();  // the round's atoms are read before the next round's
    }
}

// The force pass of sparse boxes: a warp per atom, the candidates of its 27 cells 32 at a time, the
// pairs inside the largest cutoff queued in ballot order and evaluated 32 at a time into the lanes'
// own sums, which a fixed butterfly adds.  Most cells there hold one atom or none: a warp per cell
// has little to share out, and most of its warps start for nothing.  Latency bounds it (five
// dependent loads an atom, 32 warps per SM); 100000 atoms at density 0.05 take 83 us a step, 488 with
// a warp per cell, 98 when the counts of every cell were cleared and sorted (atom_pass has more).
#define F64_ATOM_WARPS 8  // warps per block

template <bool LOG>
__global__ void __launch_bounds__(F64_ATOM_WARPS * 32) k64_force_atom(F64Args a, uint32_t step)
{
    dep_wait();
    __shared__ double4 s_qd[F64_ATOM_WARPS][F64_Q];  // queued: displacement and r^2
    __shared__ int s_qj[F64_ATOM_WARPS][F64_Q];
    const int warp = threadIdx.x >> 5;
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= a.n) return;  // warp-uniform
    const int ti = a.type[i];
    double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, bpe = 0.0, ape = 0.0;
    double vir[6] = {0, 0, 0, 0, 0, 0};
    const double rho_i = a.style == 1 ? a.rho[i] : 0.0;
    const double xi = a.x[3 * i], yi = a.x[3 * i + 1], zi = a.x[3 * i + 2];
    // lane c < 27: the c-th cell around the atom, as for a warp per cell
    int cell = 0, m = 0;
    if (lane < 27) {
        const int code = a.ccode[i];
        int cx = (code & 1023) + lane / 9 - 1, cy = ((code >> 10) & 1023) + (lane / 3) % 3 - 1,
            cz = (code >> 20) + lane % 3 - 1;
        cx += cx < 0 ? a.nc[0] : 0; cx -= cx >= a.nc[0] ? a.nc[0] : 0;
        cy += cy < 0 ? a.nc[1] : 0; cy -= cy >= a.nc[1] ? a.nc[1] : 0;
        cz += cz < 0 ? a.nc[2] : 0; cz -= cz >= a.nc[2] ? a.nc[2] : 0;
        cell = (cx * a.nc[1] + cy) * a.nc[2] + cz;
        m = min(a.cnt[cell], a.cap);
    }
    int incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const int excl = incl - m;
    const int M = __shfl_sync(0xffffffffu, incl, 31);
    const unsigned lt = (1u << lane) - 1u;
    uint32_t head = 0, tail = 0;
    auto pairs = [&](int cnt) {  // the first cnt queued pairs, one per lane
        if (lane >= cnt) return;
        const uint32_t e = (head + lane) & (F64_Q - 1);
        const double4 d = s_qd[warp][e];
        const int j = s_qj[warp][e];
        double gx, gy, gz, e2;
        if (!f64_pair(a, step, i, j, ti, d.x, d.y, d.z, d.w, a.v[3 * i] - a.v[3 * j], a.v[3 * i + 1] - a.v[3 * j + 1],
                      a.v[3 * i + 2] - a.v[3 * j + 2], rho_i, gx, gy, gz, e2))
            return;
        fx += gx;
        fy += gy;
        fz += gz;
        if (LOG) {
            pe += 0.5 * e2;
            vir[0] += 0.5 * d.x * gx; vir[1] += 0.5 * d.x * gy; vir[2] += 0.5 * d.x * gz;
            vir[3] += 0.5 * d.y * gy; vir[4] += 0.5 * d.y * gz; vir[5] += 0.5 * d.z * gz;
        }
    };
    for (int cb = 0; cb < M; cb += 32) {
        const int t = cb + lane;
        // the candidate's cell: the last of the 27 whose first record is at or before t
        // (an empty cell shares its start with the next one, which then wins)
        int c = 0;
#pragma unroll
        for (int stp = 16; stp >= 1; stp >>= 1) {
            const int probe = min(c + stp, 26);
            const int pstart = __shfl_sync(0xffffffffu, excl, probe);
            if (c + stp <= 26 && pstart <= t) c += stp;
        }
        const int cc = __shfl_sync(0xffffffffu, cell, c);
        const int c0 = __shfl_sync(0xffffffffu, excl, c);
        bool hit = false;
        double dx = 0.0, dy = 0.0, dz = 0.0, r2 = 0.0;
        int j = 0;
        if (t < M) {
            const double4 rj = a.crec[(size_t)cc * a.cap + (t - c0)];
            j = rec_index(rj);
            dx = min_image(xi - rj.x, a.L[0]);
            dy = min_image(yi - rj.y, a.L[1]);
            dz = min_image(zi - rj.z, a.L[2]);
            r2 = dx * dx + dy * dy + dz * dz;
            hit = j != i && r2 <= a.maxrc2;
        }
        const unsigned bm = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const uint32_t e = (tail + __popc(bm & lt)) & (F64_Q - 1);
            s_qd[warp][e] = make_double4(dx, dy, dz, r2);
            s_qj[warp][e] = j;
        }
        tail += __popc(bm);
        __syncwarp();
        if (tail - head >= 32u) {
            pairs(32);
            head += 32;
            __syncwarp();
        }
    }
    if (tail != head) pairs((int)(tail - head));
    f64_bonded<LOG>(a, i, lane, 32, fx, fy, fz, bpe, ape, vir);
    fx = warp_sum(fx);
    fy = warp_sum(fy);
    fz = warp_sum(fz);
    if (lane == 0) {
        a.f[3 * i] = fx;
        a.f[3 * i + 1] = fy;
        a.f[3 * i + 2] = fz;
    }
    if (LOG) {
        pe = warp_sum(pe);
        bpe = warp_sum(bpe);
        ape = warp_sum(ape);
#pragma unroll
        for (int k = 0; k < 6; k++) vir[k] = warp_sum(vir[k]);
        if (lane == 0) {
            double* q = a.q + (size_t)NQ * i;
            q[0] = pe;
            q[1] = bpe;
            q[2] = ape;
#pragma unroll
            for (int k = 0; k < 6; k++) q[3 + k] = vir[k];
        }
    }
}

// half kick and drift
__global__ void k64_initial(F64Args a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int t = a.type[i];
    if (!integrated(a, t)) return;
    const double dtm = 0.5 * a.dt / a.mass[t - 1];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        a.v[3 * i + d] += dtm * a.f[3 * i + d];
        a.x[3 * i + d] = wrap_coord(a, a.x[3 * i + d] + a.dt * a.v[3 * i + d], d, a.img + 3 * i + d);
    }
}

__global__ void k64_final(F64Args a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int t = a.type[i];
    if (!integrated(a, t)) return;
    const double dtm = 0.5 * a.dt / a.mass[t - 1];
#pragma unroll
    for (int d = 0; d < 3; d++) a.v[3 * i + d] += dtm * a.f[3 * i + d];
}

// Thermo sums in a fixed order: block b takes a contiguous range of atoms, each thread a
// fixed stride of it, then a fixed tree over the block; the final pass adds the blocks'
// partial sums in block order.  Sums: KE, m v_a v_b (6), momentum (3), pair, bond and
// angle PE, virial (6).
__global__ void __launch_bounds__(256) k64_thermo_partial(F64Args a, double* part)
{
    __shared__ double sh[NSUM][256];
    double acc[NSUM];
#pragma unroll
    for (int k = 0; k < NSUM; k++) acc[k] = 0.0;
    const int per = (a.n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per, b1 = min(a.n, b0 + per);
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        const double m = a.mass[a.type[i] - 1];
        const double vx = a.v[3 * i], vy = a.v[3 * i + 1], vz = a.v[3 * i + 2];
        acc[0] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        acc[1] += m * vx * vx; acc[2] += m * vx * vy; acc[3] += m * vx * vz;
        acc[4] += m * vy * vy; acc[5] += m * vy * vz; acc[6] += m * vz * vz;
        acc[7] += m * vx; acc[8] += m * vy; acc[9] += m * vz;
        const double* q = a.q + (size_t)NQ * i;
#pragma unroll
        for (int k = 0; k < NQ; k++) acc[10 + k] += q[k];
    }
#pragma unroll
    for (int k = 0; k < NSUM; k++) sh[k][threadIdx.x] = acc[k];
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            for (int k = 0; k < NSUM; k++) sh[k][threadIdx.x] += sh[k][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x < NSUM) part[(size_t)blockIdx.x * NSUM + threadIdx.x] = sh[threadIdx.x][0];
}

__global__ void k64_thermo_final(const double* part, int nblocks, double* sums)
{
    const int k = threadIdx.x;
    if (k >= NSUM) return;
    double s = 0.0;
    for (int b = 0; b < nblocks; b++) s += part[(size_t)b * NSUM + k];
    sums[k] = s;
}

}  // namespace

// ---------------------------------------------------------------------------------
#define F64_CK(call)                                  \
    do {                                              \
        cudaError_t e_ = (call);                      \
        if (e_ != cudaSuccess) return fail(e_, #call); \
    } while (0)

int EngineF64::fail(cudaError_t e, const char* what)
{
    err = std::string(what) + ": " + cudaGetErrorString(e);
    return DPD_E_CUDA;
}

EngineF64::~EngineF64()
{
    void* ptrs[] = {x_, v_, xn_, vn_, cnt_next_, owner_, owner_prev_, f_, rho_, q_, part_, sums_, img_, type_, cnt_, ccode_, craw_, crec_, status_,
                    bstart_, astart_, bent_, aent_, tab_};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (stream_) cudaStreamDestroy(stream_);
}

template <class T>
static cudaError_t dalloc64(T** p, size_t n, int64_t& bytes)
{
    bytes += (int64_t)(sizeof(T) * (n ? n : 1));
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * (n ? n : 1));
    if (e == cudaSuccess) e = cudaMemset(*p, 0, sizeof(T) * (n ? n : 1));
    return e;
}

// cells that hold an atom of the input (an atom without a position, an error later, counts nowhere)
int EngineF64::occupied_cells() const
{
    std::vector<char> seen((size_t)ncell_, 0);
    int count = 0;
    for (int i = 0; i < n_; i++) {
        size_t cell = 0;
        for (int d = 0; d < 3; d++) {
            double q = (R_.sys.x[3 * (size_t)i + d] - R_.sys.lo[d]) / L_[d];
            if (!std::isfinite(q)) {
                cell = (size_t)ncell_;
                break;
            }
            q -= std::floor(q);
            cell = cell * nc_[d] + std::min((int)(q * nc_[d]), nc_[d] - 1);
        }
        if (cell < (size_t)ncell_ && !seen[cell]) {
            seen[cell] = 1;
            count++;
        }
    }
    return count;
}

int EngineF64::init(Replica&& rep)
{
    R_ = std::move(rep);
    const RunInput& in = R_.in;
    const ForceField& ff = R_.ff;
    // the parity mode covers the force field and NVE; every fix and compute other than
    // nve, and dumps, belong to the single-precision engine
    if (ff.spring.on || ff.rvcm.on || ff.recenter.on || !ff.moves.empty() || !ff.reflects.empty() ||
        !ff.twowalls.empty() || !ff.gcs.empty() || !ff.cdumps.empty() || !ff.rdfs.empty() || in.dump) {
        err = "the FP64 parity mode runs pair, bond and angle styles with fix nve only: "
              "remove the other fixes, computes and dumps";
        return DPD_E_ARG;
    }
    if (in.log_f == 0) {
        err = "thermo interval must be positive";
        return DPD_E_ARG;
    }
    n_ = R_.sys.n_atoms;
    if (n_ < 2) {
        err = "the FP64 parity mode needs at least 2 atoms";
        return DPD_E_ARG;
    }
    for (int d = 0; d < 3; d++) {
        L_[d] = R_.sys.hi[d] - R_.sys.lo[d];
        nc_[d] = (int)std::floor(L_[d] / in.global_cut);
        if (nc_[d] < 3) {
            err = "box too small: the cell grid needs at least 3 cells of size global_cut per dimension";
            return DPD_E_ARG;
        }
        if (nc_[d] > DPD_MAX_NC) {
            err = "box too large: at most 1023 cells per dimension";
            return DPD_E_ARG;
        }
    }
    ncell_ = nc_[0] * nc_[1] * nc_[2];
    const double wv = (L_[0] / nc_[0]) * (L_[1] / nc_[1]) * (L_[2] / nc_[2]);
    cap_ = std::max(32, (((int)(2.0 * in.max_rho * wv) + 1 + 15) / 16) * 16);
    // every table index the kernels take from the input is checked here
    const int ntyp = R_.sys.n_atomtypes;
    const int nbtyp = std::max(R_.sys.n_bondtypes, 1), natyp = std::max(R_.sys.n_angletypes, 1);
    if ((int)R_.sys.type.size() < n_ || (int)R_.sys.masses.size() < ntyp ||
        (int)ff.coeff.size() < ntyp * (ntyp + 1) / 2) {
        err = "incomplete system or pair coefficients";
        return DPD_E_ARG;
    }
    for (int i = 0; i < n_; i++)
        if (R_.sys.type[i] < 1 || R_.sys.type[i] > ntyp) {
            err = "atom type out of range";
            return DPD_E_ARG;
        }
    // bonds and angles in tag order, as adjacency lists of each atom
    const int nb = R_.sys.n_bonds, na = R_.ff.angle_style ? R_.sys.n_angles : 0;
    for (int b = 0; b < nb; b++)
        if (R_.sys.bonds[3 * b] < 1 || R_.sys.bonds[3 * b] > nbtyp) {
            err = "bond type out of range";
            return DPD_E_ARG;
        }
    for (int t = 0; t < na; t++)
        if (R_.sys.angles[4 * t] < 1 || R_.sys.angles[4 * t] > natyp) {
            err = "angle type out of range";
            return DPD_E_ARG;
        }
    std::vector<int> bstart(n_ + 1, 0), astart(n_ + 1, 0);
    auto tag_ok = [&](int t) { return t >= 1 && t <= n_; };
    for (int b = 0; b < nb; b++) {
        const int* e = &R_.sys.bonds[3 * b];
        if (!tag_ok(e[1]) || !tag_ok(e[2])) {
            err = "bond partner not found";
            return DPD_E_STATE;
        }
        bstart[e[1]]++;
        bstart[e[2]]++;
    }
    for (int t = 0; t < na; t++) {
        const int* e = &R_.sys.angles[4 * t];
        if (!tag_ok(e[1]) || !tag_ok(e[2]) || !tag_ok(e[3])) {
            err = "angle atom not found";
            return DPD_E_STATE;
        }
        astart[e[1]]++;
        astart[e[2]]++;
        astart[e[3]]++;
    }
    for (int i = 0; i < n_; i++) {
        bstart[i + 1] += bstart[i];
        astart[i + 1] += astart[i];
    }
    std::vector<int2> bent(std::max(2 * nb, 1));
    std::vector<int4> aent(std::max(3 * na, 1));
    {
        std::vector<int> fb(bstart.begin(), bstart.end() - 1), fa(astart.begin(), astart.end() - 1);
        for (int b = 0; b < nb; b++) {
            const int* e = &R_.sys.bonds[3 * b];
            const int i = e[1] - 1, j = e[2] - 1;
            bent[fb[i]++] = make_int2(j, e[0]);
            bent[fb[j]++] = make_int2(i, e[0]);
        }
        for (int t = 0; t < na; t++) {
            const int* e = &R_.sys.angles[4 * t];
            const int4 an = make_int4(e[1] - 1, e[2] - 1, e[3] - 1, e[0]);
            for (int k = 1; k <= 3; k++) aent[fa[e[k] - 1]++] = an;
        }
    }
    // coefficient tables
    const int nt = R_.sys.n_atomtypes, ntri = nt * (nt + 1) / 2;
    const int nbt = std::max(R_.sys.n_bondtypes, 1), nat = std::max(R_.sys.n_angletypes, 1);
    std::vector<double> tab((size_t)NC * ntri + nt + 4 * nbt + 2 * nat, 0.0);
    // sqrt(2 kT) / sqrt(dt), src/force/pair_dpd.cu:577-578
    const double sig_scale = std::sqrt(2.0 * ff.temp) / std::sqrt(in.dt);
    for (int p = 0; p < ntri && p < (int)ff.coeff.size(); p++) {
        double* c = &tab[(size_t)NC * p];
        for (int k = 0; k < 5; k++) c[k] = ff.coeff[p][k];
        c[5] = std::sqrt(c[2]) * sig_scale;
        c[6] = c[3] > 0.0 ? 1.0 / c[3] : 0.0;
        c[7] = c[4] > 0.0 ? 1.0 / c[4] : HUGE_VAL;  // no rd: w_d clamps to 0
        c[8] = c[3] * c[3];
    }
    for (int t = 0; t < nt; t++) tab[NC * ntri + t] = R_.sys.masses[t];
    for (int b = 0; b < (int)ff.bond_coeff.size() && b < nbt; b++)
        for (int k = 0; k < 4; k++) tab[NC * ntri + nt + 4 * b + k] = ff.bond_coeff[b][k];
    for (int b = 0; b < (int)ff.angle_coeff.size() && b < nat; b++)
        for (int k = 0; k < 2; k++) tab[NC * ntri + nt + 4 * nbt + 2 * b + k] = ff.angle_coeff[b][k];

    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        err = "no CUDA device available (this engine has no CPU fallback)";
        return DPD_E_NODEV;
    }
    if (const char* dv = std::getenv("DPD_B200_DEVICE")) {  // as the single-precision engine
        const int dev = std::atoi(dv);
        if (dev < 0 || dev >= ndev) {
            err = "DPD_B200_DEVICE is not a device index";
            return DPD_E_NODEV;
        }
        F64_CK(cudaSetDevice(dev));
    }
    F64_CK(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    const size_t n = (size_t)n_;
    F64_CK(dalloc64(&x_, 3 * n, bytes_));
    F64_CK(dalloc64(&v_, 3 * n, bytes_));
    F64_CK(dalloc64(&f_, 3 * n, bytes_));
    F64_CK(dalloc64(&rho_, n, bytes_));
    F64_CK(dalloc64(&q_, (size_t)NQ * n, bytes_));
    F64_CK(dalloc64(&part_, (size_t)NSUM * RED_BLOCKS, bytes_));
    F64_CK(dalloc64(&sums_, (size_t)NSUM, bytes_));
    F64_CK(dalloc64(&img_, 3 * n, bytes_));
    F64_CK(dalloc64(&type_, n, bytes_));
    F64_CK(dalloc64(&cnt_, (size_t)ncell_, bytes_));
    F64_CK(dalloc64(&cnt_next_, (size_t)ncell_, bytes_));
    // the occupied cells are counted where they can matter: min(n, ncell) is the most there can be
    const int most = std::min(n_, ncell_);
    const int occupied = atom_pass(n_, ncell_, most) || atom_pass_logged(n_, most) ? occupied_cells() : most;
    sparse_ = atom_pass(n_, ncell_, occupied);
    log_by_atom_ = sparse_ || atom_pass_logged(n_, occupied);
    if (sparse_) {
        F64_CK(dalloc64(&owner_, n, bytes_));
        F64_CK(dalloc64(&owner_prev_, n, bytes_));
    } else {
        F64_CK(dalloc64(&xn_, 3 * n, bytes_));
        F64_CK(dalloc64(&vn_, 3 * n, bytes_));
        F64_CK(dalloc64(&craw_, (size_t)ncell_ * cap_, bytes_));
    }
    F64_CK(dalloc64(&ccode_, n, bytes_));
    F64_CK(dalloc64(&crec_, (size_t)ncell_ * cap_, bytes_));
    F64_CK(dalloc64(&status_, 1, bytes_));
    F64_CK(dalloc64(&bstart_, n + 1, bytes_));
    F64_CK(dalloc64(&astart_, n + 1, bytes_));
    F64_CK(dalloc64(&bent_, bent.size(), bytes_));
    F64_CK(dalloc64(&aent_, aent.size(), bytes_));
    F64_CK(dalloc64(&tab_, tab.size(), bytes_));
    F64_CK(cudaMemcpy(type_, R_.sys.type.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    F64_CK(cudaMemcpy(bstart_, bstart.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice));
    F64_CK(cudaMemcpy(astart_, astart.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice));
    F64_CK(cudaMemcpy(bent_, bent.data(), sizeof(int2) * bent.size(), cudaMemcpyHostToDevice));
    F64_CK(cudaMemcpy(aent_, aent.data(), sizeof(int4) * aent.size(), cudaMemcpyHostToDevice));
    F64_CK(cudaMemcpy(tab_, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice));
    return upload_state(true, true);
}

// positions wrapped into [lo, lo + L) with image counts from zero (as a data file is
// read) and/or velocities; the next run starts with a zero step
int EngineF64::upload_state(bool pos, bool vel)
{
    const size_t n3 = 3 * (size_t)n_;
    zero_pending_ = true;
    if (vel) {
        std::vector<double> v(n3, 0.0);
        if (R_.sys.v.size() >= n3) std::copy(R_.sys.v.begin(), R_.sys.v.begin() + n3, v.begin());
        F64_CK(cudaMemcpyAsync(v_, v.data(), sizeof(double) * n3, cudaMemcpyHostToDevice, stream_));
        F64_CK(cudaStreamSynchronize(stream_));
    }
    if (!pos) return DPD_OK;
    std::vector<double> x(R_.sys.x.begin(), R_.sys.x.begin() + n3);
    std::vector<int> img(n3, 0);
    for (size_t k = 0; k < n3; k++) {
        const int d = (int)(k % 3);
        double p = x[k];
        if (!std::isfinite(p)) {
            err = "non-finite position in the input";
            return DPD_E_ARG;
        }
        const double lo = R_.sys.lo[d], hi = lo + L_[d];
        if (p >= hi || p < lo) {
            const double q = std::floor((p - lo) / L_[d]);
            p -= L_[d] * q;
            img[k] += (int)q;
            if (p >= hi) p = lo;
            if (p < lo) p = lo;
        }
        x[k] = p;
    }
    F64_CK(cudaMemcpyAsync(x_, x.data(), sizeof(double) * n3, cudaMemcpyHostToDevice, stream_));
    F64_CK(cudaMemcpyAsync(img_, img.data(), sizeof(int) * n3, cudaMemcpyHostToDevice, stream_));
    F64_CK(cudaStreamSynchronize(stream_));
    return DPD_OK;
}

static F64Args make_args(const Replica& R, int n, const int nc[3], const double L[3], int cap)
{
    F64Args a;
    memset(&a, 0, sizeof(a));
    a.n = n;
    a.ntypes = R.sys.n_atomtypes;
    a.style = R.ff.pair_style;
    a.bond_style = R.sys.n_bonds > 0 ? R.ff.bond_style : 0;
    a.angle_style = R.ff.angle_style;
    a.cap = cap;
    a.seed = R.ff.seed;
    a.integ_mask = R.ff.integ_mask;
    a.dt = R.in.dt;
    double rcm = 0.0;
    for (auto& c : R.ff.coeff) rcm = std::max(rcm, c[3]);
    a.maxrc2 = rcm * rcm;
    for (int d = 0; d < 3; d++) {
        a.nc[d] = nc[d];
        a.lo[d] = R.sys.lo[d];
        a.L[d] = L[d];
        a.w[d] = L[d] / nc[d];
    }
    return a;
}

// the launch may overlap the tail of its predecessor (the kernel starts with dep_wait)
template <typename... KArgs, typename... Args>
static void launch_dep(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// The forces of a step from the current positions and velocities.  binned: the previous step
// has put the atoms into their cells; advance: the force pass also takes them to the next
// step's positions and cells (steps without thermo), and the buffers change places.
int EngineF64::eval_forces(uint32_t step, bool log, bool binned, bool advance)
{
    F64Args a = make_args(R_, n_, nc_, L_, cap_);
    const int nt = R_.sys.n_atomtypes, ntri = nt * (nt + 1) / 2, nbt = std::max(R_.sys.n_bondtypes, 1);
    a.coeff = tab_;
    a.mass = tab_ + NC * ntri;
    a.bondc = tab_ + NC * ntri + nt;
    a.anglec = tab_ + NC * ntri + nt + 4 * nbt;
    a.x = x_; a.v = v_; a.f = f_; a.rho = rho_; a.q = q_; a.xn = xn_; a.vn = vn_;
    a.img = img_; a.type = type_; a.cnt = cnt_; a.cnt_next = cnt_next_; a.craw = craw_; a.crec = crec_;
    a.status = status_; a.ccode = ccode_; a.owner = owner_; a.owner_prev = owner_prev_;
    a.bstart = bstart_; a.astart = astart_; a.bent = bent_; a.aent = aent_;
    const int gw = (int)(((size_t)n_ * 32 + 255) / 256);  // a warp per atom
    const int g = (n_ + 255) / 256;
    if (sparse_) k64_bin_owned<<<g, 256, 0, stream_>>>(a);
    else if (!binned) k64_bin<<<g, 256, 0, stream_>>>(a);
    if (sparse_) launch_dep(k64_sort_owned, g, 256, 0, stream_, a);
    else launch_dep(k64_sort_cells, (int)(((size_t)ncell_ * 8 + 255) / 256), 256, 0, stream_, a, ncell_);
    if (a.style == 1) launch_dep(k64_density, gw, 256, 0, stream_, a);
    const int gf = (ncell_ + F64_WARPS - 1) / F64_WARPS, tf = F64_WARPS * 32;  // a warp per cell
    const int ga = (n_ + F64_ATOM_WARPS - 1) / F64_ATOM_WARPS, ta = F64_ATOM_WARPS * 32;  // a warp per atom
    if (log && log_by_atom_) launch_dep(k64_force_atom<true>, ga, ta, 0, stream_, a, step);
    else if (sparse_) launch_dep(k64_force_atom<false>, ga, ta, 0, stream_, a, step);
    else if (log) launch_dep(k64_force<true, false>, gf, tf, F64_WARPS * sizeof(F64Warp<true>), stream_, a, step, ncell_);
    else if (!advance)
        launch_dep(k64_force<false, false>, gf, tf, F64_WARPS * sizeof(F64Warp<false>), stream_, a, step, ncell_);
    else {
        launch_dep(k64_force<false, true>, gf, tf, F64_WARPS * sizeof(F64Warp<false>), stream_, a, step, ncell_);
        std::swap(x_, xn_);
        std::swap(v_, vn_);
    }
    // the sort has cleared the other counts: the next binning fills them
    std::swap(cnt_, cnt_next_);
    std::swap(owner_, owner_prev_);
    F64_CK(cudaGetLastError());
    return DPD_OK;
}

// the thermo row of a logged step (src/compute/thermo.cu): T = 2 KE / (3N - 3),
// P_ab = (sum m v_a v_b + W_ab) / V, P = trace / 3
int EngineF64::log_row(uint32_t step)
{
    F64Args a = make_args(R_, n_, nc_, L_, cap_);
    const int nt = R_.sys.n_atomtypes, ntri = nt * (nt + 1) / 2;
    a.mass = tab_ + NC * ntri;
    a.v = v_; a.q = q_; a.type = type_;
    const int nb = std::min((int)RED_BLOCKS, (n_ + 255) / 256);
    k64_thermo_partial<<<nb, 256, 0, stream_>>>(a, part_);
    k64_thermo_final<<<1, 32, 0, stream_>>>(part_, nb, sums_);
    double s[NSUM];
    F64_CK(cudaMemcpyAsync(s, sums_, sizeof(s), cudaMemcpyDeviceToHost, stream_));
    F64_CK(cudaStreamSynchronize(stream_));
    dpd_thermo t;
    memset(&t, 0, sizeof(t));
    const double vol = L_[0] * L_[1] * L_[2];
    t.step = step;
    t.ke = s[0];
    t.temp = 2.0 * s[0] / (3.0 * n_ - 3.0);
    t.pair_pe = s[10];
    t.bond_pe = s[11];
    t.angle_pe = s[12];
    for (int c = 0; c < 6; c++) t.p[c] = (s[1 + c] + s[13 + c]) / vol;
    t.pressure = (t.p[0] + t.p[3] + t.p[5]) / 3.0;
    for (int c = 0; c < 3; c++) t.momentum[c] = s[7 + c];
    rows_.push_back(t);
    return DPD_OK;
}

int EngineF64::check_status()
{
    int st = 0;
    F64_CK(cudaMemcpyAsync(&st, status_, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    F64_CK(cudaStreamSynchronize(stream_));
    if (st & F64_CELL_OVERFLOW) {
        err = "cell overflow in the FP64 parity mode: increase max_rho in the neighbor command";
        return DPD_E_OVERFLOW;
    }
    if (st & (F64_NONFINITE | F64_FAR)) {
        err = "non-finite position or velocity";
        return DPD_E_NUMERIC;
    }
    if (st & F64_FENE) {
        err = "FENE bond stretched beyond R0";
        return DPD_E_NUMERIC;
    }
    return DPD_OK;
}

// Steps in the order of the reference's loop (src/main/utils.cuh:166-213 for the zero
// step, :254-303 per step): the zero step evaluates forces at the current step and logs
// it when due; each step then kicks and drifts, evaluates forces, kicks, and logs.
int EngineF64::run(uint32_t nsteps)
{
    F64Args a = make_args(R_, n_, nc_, L_, cap_);
    const int nt = R_.sys.n_atomtypes, ntri = nt * (nt + 1) / 2;
    a.mass = tab_ + NC * ntri;
    a.f = f_; a.img = img_; a.type = type_; a.status = status_;
    const int g = (n_ + 255) / 256;
    const uint32_t log_f = R_.in.log_f;
    int e;
    if (zero_pending_) {
        const uint32_t s0 = next_step_;
        const bool log = s0 % log_f == 0;
        if ((e = eval_forces(s0, log, false, false))) return e;
        if ((e = check_status())) return e;
        if (log && (e = log_row(s0))) return e;
        zero_pending_ = false;
        next_step_ = s0 + 1;
    }
    bool binned = false;  // the previous step's force pass has already drifted and binned the atoms
    for (uint32_t k = 0; k < nsteps; k++) {
        const uint32_t step = next_step_;
        const bool log = step % log_f == 0, advance = !log && !sparse_ && k + 1 < nsteps;
        a.x = x_;
        a.v = v_;
        if (!binned) k64_initial<<<g, 256, 0, stream_>>>(a);
        if ((e = eval_forces(step, log, binned, advance))) return e;
        binned = advance;
        if (!advance) {
            k64_final<<<g, 256, 0, stream_>>>(a);
            F64_CK(cudaGetLastError());
        }
        if (log) {
            if ((e = log_row(step))) return e;
            if ((e = check_status())) return e;
        }
        next_step_ = step + 1;
    }
    return check_status();
}

int EngineF64::get_thermo(dpd_thermo* rows, int max_rows, int* n_rows) const
{
    const int n = std::min((int)rows_.size(), std::max(max_rows, 0));
    for (int k = 0; k < n; k++) rows[k] = rows_[rows_.size() - n + k];
    if (n_rows) *n_rows = n;
    return DPD_OK;
}

int EngineF64::get_state(double* x, double* v, int* image, double* f)
{
    const size_t n3 = 3 * (size_t)n_;
    if (x) F64_CK(cudaMemcpyAsync(x, x_, sizeof(double) * n3, cudaMemcpyDeviceToHost, stream_));
    if (v) F64_CK(cudaMemcpyAsync(v, v_, sizeof(double) * n3, cudaMemcpyDeviceToHost, stream_));
    if (image) F64_CK(cudaMemcpyAsync(image, img_, sizeof(int) * n3, cudaMemcpyDeviceToHost, stream_));
    if (f) F64_CK(cudaMemcpyAsync(f, f_, sizeof(double) * n3, cudaMemcpyDeviceToHost, stream_));
    F64_CK(cudaStreamSynchronize(stream_));
    return DPD_OK;
}

// nsteps steps timed with CUDA events on the engine's stream
int EngineF64::time_steps(uint32_t nsteps, double* total_ms)
{
    if (zero_pending_) {
        int e = run(0);
        if (e) return e;
    }
    cudaEvent_t e0, e1;
    F64_CK(cudaEventCreate(&e0));
    F64_CK(cudaEventCreate(&e1));
    F64_CK(cudaEventRecord(e0, stream_));
    int e = run(nsteps);
    cudaEventRecord(e1, stream_);
    cudaEventSynchronize(e1);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e) return e;
    if (total_ms) *total_ms = ms;
    return DPD_OK;
}

// the reference's write_data file of the current state (as the single-precision engine)
int EngineF64::write_data(const std::string& path)
{
    SystemData s = R_.sys;
    s.v.resize(s.x.size());
    int e = get_state(s.x.data(), s.v.data(), nullptr, nullptr);
    if (e) return e;
    return write_data_file(path, R_.in.atom_style, s, err);
}

// new positions (image counts restart from zero) and/or velocities by tag; the next run
// starts with a zero step
int EngineF64::set_state(const double* x, const double* v)
{
    const size_t n3 = 3 * (size_t)n_;
    if (x) std::copy(x, x + n3, R_.sys.x.begin());
    if (v) {
        R_.sys.v.resize(n3);
        std::copy(v, v + n3, R_.sys.v.begin());
    }
    return upload_state(x != nullptr, v != nullptr);
}

}  // namespace dpd
