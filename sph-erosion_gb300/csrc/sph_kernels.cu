// Hand-written sm_103a kernels of one simulation step, all scenes of a system
// per launch.  Work is a list of (scene, tile) items: a block per tile, which
// the hardware hands to SMs as they free up; warps that take slices of tiles
// from a counter (the force pass over lists); or, in small systems, a group of
// lanes per particle of a tile.  A scene whose step budget is exhausted is
// skipped.
//
// Stage order per step (the reference's Run, Erosion/fluid_system.h:104-183,
// with its three O(N^2) passes replaced by a uniform grid):
//   keys -> scan -> scatter -> reorder   counting sort into Morton-ordered cell rows along x;
//                                         one kernel where every scene is small (sort_small_smem)
//   density                               pass 1 (:107-124)
//   force                                 passes 2 and 3 (:127-178), advance
//                                         (:306-353), box (:355-407), terrain
//                                         contact and erosion exchange
//   terrain                               height snapshot for the next step
//
// Every arithmetic operation of the physics uses an explicitly rounded
// intrinsic (__fmul_rn, __fadd_rn, ...), which the compiler never contracts
// into a fused multiply-add, so each term rounds exactly like the reference's
// scalar FP32 code.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sph_kernels.h"

namespace sph {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// The kernels of a step follow one another on one stream and each needs all of
// the one before.  In small systems those that launch() starts early may come
// to the SMs while the kernel before them runs, and wait here until it has
// completed and its writes are visible.  Every thread of such a kernel calls
// this first.  Only then does the kernel let its own dependent start: a
// dependent is resident beside the one kernel it waits for and never beside an
// earlier one, whose reads could leave old lines in an L1 that its own reads
// meet.  While it waits, that kernel writes what it will read, so it takes none
// of the step's arrays through the non-coherent path (__ldg), which requires
// them to be constant for a kernel's whole life; the row table is, since only
// copies write it.
__device__ __forceinline__ void step_enter(bool early) {
    if (!early) return;  // not launched that way: the instructions are not free (terrain kernel 31 vs 21 us)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fsq(float a) { return __fsqrt_rn(a); }

// x^2 with one rounding (what a correctly rounded powf(x, 2.0f) returns).
__device__ __forceinline__ float pow2(float x) { return __fmul_rn(x, x); }

// x^3 rounded once in all but near-tie cases: x*x = p + e exactly and
// p*x = c + f exactly (TwoProduct with FMA; Ogita, Rump and Oishi, "Accurate
// sum and dot product", SIAM J. Sci. Comput. 2005), then c + (f + e*x).
__device__ __forceinline__ float pow3(float x) {
    float p = __fmul_rn(x, x);
    float e = __fmaf_rn(x, x, -p);
    float c = __fmul_rn(p, x);
    float f = __fmaf_rn(p, x, -c);
    float t = __fmaf_rn(e, x, f);
    return __fadd_rn(c, t);
}

// Squared distance of the reference's glm::length, (dx*dx + dy*dy) + dz*dz.
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
    return fa(fa(fm(dx, dx), fm(dy, dy)), fm(dz, dz));
}

// Two floats in one 64-bit register pair and the packed FP32 operations on
// them (sm_100 and later): one instruction for two operations, each half
// rounded like its scalar form, so they change no bits.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 pk(float v) { return pk(v, v); }
__device__ __forceinline__ float lo(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) { return fma2(a, pk(1.0f), b); }
// A product that an addition follows, as a * b + (-0) with a -0 that the
// assembler does not know (neg_zero, read once per kernel): it fuses
// mul.rn.f32x2 into an addition that uses its result (also into a scalar one),
// which would drop the product's rounding; this form it cannot fuse.
__constant__ float kNegZero = -0.0f;
__device__ __forceinline__ f2 neg_zero() { return pk(*(volatile const float*)&kNegZero); }
__device__ __forceinline__ f2 mulr2(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }

// A packed neighbour record (DevArrays::fdat) as four pairs: (x, y),
// (z, P/rho^2), (vx, vy), (vz, m/rho); one 256-bit load.
struct Rec {
    f2 xy, zA, vxy, vzB;
};
__device__ __forceinline__ Rec ld_rec(const float4* p) {
    Rec r;
    asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(r.xy), "=l"(r.zA), "=l"(r.vxy), "=l"(r.vzB) : "l"(p));
    return r;
}

__device__ __forceinline__ int cell_coord(float x, float lo, float inv, int n) {
    float t = fm(fs(x, lo), inv);
    if (!(t > 0.0f)) t = 0.0f;  // also maps NaN to 0
    float top = (float)(n - 1);
    if (t > top) t = top;
    return (int)t;
}

struct Cell {
    int cx, cy, cz;
};

__device__ __forceinline__ Cell cell_of(const SceneDev& S, float x, float y, float z) {
    Cell c;
    c.cx = cell_coord(x, S.lo[0], S.inv_cell_x, S.nx);
    c.cy = cell_coord(y, S.lo[1], S.inv_cell, S.ny);
    c.cz = cell_coord(z, S.lo[2], S.inv_cell, S.nz);
    return c;
}

__device__ __forceinline__ uint32_t row_key(const uint32_t* tab, const SceneDev& S, int cy, int cz) {
    return __ldg(tab + S.tab_off + cz * S.ny + cy) * (uint32_t)S.nx;
}

// A particle's position in cell units before flooring and clamping, and its
// cell.
struct Probe {
    Cell c;
    float tx, ty, tz;
    bool finite;
};

__device__ __forceinline__ Probe probe_of(const SceneDev& S, float4 x) {
    Probe q;
    q.tx = fm(fs(x.x, S.lo[0]), S.inv_cell_x);
    q.ty = fm(fs(x.y, S.lo[1]), S.inv_cell);
    q.tz = fm(fs(x.z, S.lo[2]), S.inv_cell);
    q.finite = (q.tx == q.tx) && (q.ty == q.ty) && (q.tz == q.tz);
    q.c = cell_of(S, x.x, x.y, x.z);
    return q;
}

// Distance in cell units from coordinate t to cell k of an axis of n cells.
// The two end cells reach to infinity: positions outside the grid are
// clamped into them.
__device__ __forceinline__ float cell_gap(float t, int k, int n) {
    float g = 0.0f;
    if (k > 0 && t < (float)k) g = (float)k - t;
    if (k < n - 1 && t > (float)(k + 1)) g = t - (float)(k + 1);
    return g;
}

// Cells [xl, xh] of row (y, z) that the h-sphere around the particle can
// reach; false when it reaches none.  Conservative (h enlarged by hcell's
// slack), so only out-of-range candidates are ever dropped and the in-range
// visiting order is the same as for the full (2R+1)^3 block.
__device__ __forceinline__ bool row_span(const SceneDev& S, const Probe& q, int y, int z, int* xl, int* xh) {
    if (!q.finite) return false;  // a NaN position has no neighbour, itself included
    const float gy = cell_gap(q.ty, y, S.ny), gz = cell_gap(q.tz, z, S.nz);
    const float r2 = S.hcell * S.hcell - gy * gy - gz * gz;
    if (!(r2 >= 0.0f)) return false;
    const float r = sqrtf(r2) * (float)S.xsub;  // in x cells
    const float top = (float)(S.nx - 1);
    const float lo = fminf(fmaxf(floorf(q.tx - r), 0.0f), top);
    const float hi = fminf(fmaxf(floorf(q.tx + r), 0.0f), top);
    *xl = (int)lo;
    *xh = (int)hi;
    return true;
}

// Cell rows of the neighbour search.  for_rows(a, S, xi, valid, fn) calls
// fn(st, en) for each of the (2R+1)^2 rows (dz outer, dy inner, both
// ascending) with the particle range [st, en) of the row's cells that the
// h-sphere around xi can reach; a row it cannot reach (or any row when
// valid is false) gives an empty range, so every lane makes the same calls.
// The reach test is conservative (h enlarged by hcell's slack): only
// out-of-range candidates are ever dropped and the in-range visiting order is
// that of the full (2R+1)^3 block.
//
// At reach 1 (cells of h or more) cells along x are half as long as along y
// and z (xsub 2): a row's range is trimmed to the sphere in finer steps at
// no extra row.  For R = 1 and 2 (y/z cells of h and h/2, x reach 2 cells
// either way) the squared gaps of the 5 x cells are computed once per
// particle (registers), so a row costs a few adds and compares; the row loops stay rolled to keep register pressure (and
// so occupancy) where these latency-bound kernels need it.  Other reaches
// take the general path.
template <int R, class Fn>
__device__ __forceinline__ void for_rows_r(const DevArrays& a, const SceneDev& S, float4 xi, bool valid, Fn&& fn) {
    const Probe q = probe_of(S, xi);
    const uint32_t* off = a.offsets + S.k_off;
    const uint32_t* tab = a.tab + S.tab_off;
    const float H2 = S.hcell * S.hcell;
    constexpr int XS = R == 1 ? 2 : 1;  // the scene's xsub at this reach
    constexpr int RX = R * XS;          // reach along x, in x cells
    float gx2[2 * RX + 1];              // squared x-gaps in y/z cell units
#pragma unroll
    for (int d = -RX; d <= RX; ++d) {
        const int k = q.c.cx + d;
        float g2 = INFINITY;
        if (k >= 0 && k < S.nx) {
            const float g = cell_gap(q.tx, k, S.nx) * (1.0f / XS);
            g2 = g * g;
        }
        gx2[d + RX] = g2;
    }
    const bool live = valid && q.finite;
#pragma unroll 1
    for (int dz = -R; dz <= R; ++dz) {
        const int z = q.c.cz + dz;
        const bool zin = live && z >= 0 && z < S.nz;
        float gz2 = INFINITY;
        const uint32_t* tz = tab + (zin ? z : 0) * S.ny;  // row numbers of slab z
        if (zin) {
            const float g = cell_gap(q.tz, z, S.nz);
            gz2 = g * g;
        }
#pragma unroll 1
        for (int dy = -R; dy <= R; ++dy) {
            const int y = q.c.cy + dy;
            uint32_t st = 0, en = 0;
            if (zin && y >= 0 && y < S.ny) {
                const float g = cell_gap(q.ty, y, S.ny);
                const float r2 = H2 - g * g - gz2;
                if (r2 >= 0.0f) {
                    int lo = 0, hi = 0;  // farthest reachable cell on each side
#pragma unroll
                    for (int d = 1; d <= RX; ++d) {
                        if (gx2[RX - d] <= r2) lo = -d;
                        if (gx2[RX + d] <= r2) hi = d;
                    }
                    const uint32_t row = __ldg(tz + y) * (uint32_t)S.nx;
                    st = __ldg(off + row + q.c.cx + lo);
                    en = __ldg(off + row + q.c.cx + hi + 1);
                }
            }
            fn(st, en);
        }
    }
}

template <class Fn>
__device__ __forceinline__ void for_rows_any(const DevArrays& a, const SceneDev& S, float4 xi, bool valid, Fn&& fn) {
    const Probe q = probe_of(S, xi);
    const int R = S.reach;
    const uint32_t* off = a.offsets + S.k_off;
    for (int dz = -R; dz <= R; ++dz) {
        for (int dy = -R; dy <= R; ++dy) {
            const int z = q.c.cz + dz, y = q.c.cy + dy;
            uint32_t st = 0, en = 0;
            int xl, xh;
            if (valid && z >= 0 && z < S.nz && y >= 0 && y < S.ny && row_span(S, q, y, z, &xl, &xh)) {
                const uint32_t row = row_key(a.tab, S, y, z);
                st = __ldg(off + row + xl);
                en = __ldg(off + row + xh + 1);
            }
            fn(st, en);
        }
    }
}

template <class Fn>
__device__ __forceinline__ void for_rows(const DevArrays& a, const SceneDev& S, float4 xi, bool valid, Fn&& fn) {
    if (S.reach == 2)
        for_rows_r<2>(a, S, xi, valid, fn);
    else if (S.reach == 1)
        for_rows_r<1>(a, S, xi, valid, fn);
    else
        for_rows_any(a, S, xi, valid, fn);
}

// Visit every candidate of the trimmed rows around xi: f(j, xj) receives the
// scene-local sorted index and the position.
template <class F>
__device__ __forceinline__ void for_each_candidate(const DevArrays& a, const SceneDev& S, float4 xi, F&& f) {
    const float4* sp = a.spos + S.p_off;
    for_rows(a, S, xi, true, [&](uint32_t st, uint32_t en) {
        for (uint32_t j = st; j < en; ++j) f(j, __ldg(sp + j));
    });
}

// In-range traversal of the fast path.  Candidates are tested in a tight
// loop and the indices of in-range ones are compacted into a per-thread list
// in shared memory (column threadIdx.x, so lanes touch distinct banks); the
// costly pair terms then run over the list with every lane of the warp busy
// instead of diverging on each candidate.  The visiting order is the
// candidate order, so the sums are the same as a direct traversal.
//
// All lanes of a warp visit the same (dz, dy) cell row at the same time and
// step through it for the longest lane's length, so the list drain is a
// collective step: it runs as soon as any lane's list is full, with all lanes
// draining theirs.  Every lane of the warp must call this function (lanes
// without a particle pass valid = false).
constexpr int kListCap = 32;

template <class F>
__device__ __forceinline__ void for_each_in_range_listed(const DevArrays& a, const SceneDev& S, bool valid,
                                                         float4 xi, uint32_t* list, F&& f) {
    const float4* sp = a.spos + S.p_off;
    uint32_t* my = list + threadIdx.x;
    const int stride = blockDim.x;
    int cnt = 0;
    for_rows(a, S, xi, valid, [&](uint32_t st, uint32_t en) {
        const uint32_t len = en - st;
        const uint32_t maxlen = __reduce_max_sync(kFull, len);
        for (uint32_t t = 0; t < maxlen; ++t) {
            if (t < len) {
                const uint32_t j = st + t;
                const float4 xj = __ldg(sp + j);
                const float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                if (s <= S.smax) my[(cnt++) * stride] = j;
            }
            if (__any_sync(kFull, cnt == kListCap)) {
                for (int q = 0; q < cnt; ++q) f(my[q * stride]);
                cnt = 0;
            }
        }
    });
    for (int q = 0; q < cnt; ++q) f(my[q * stride]);
}

// Ordered (validation) traversal: collect in-range candidates, sort them by
// particle id and visit them in ascending id, which is the reference's
// summation order (all j ascending).
constexpr int kMaxNb = 128;

template <class F>
__device__ __forceinline__ bool for_each_in_range_ordered(const DevArrays& a, const SceneDev& S, float4 xi,
                                                           F&& f) {
    unsigned long long lst[kMaxNb];
    int cnt = 0;
    bool overflow = false;
    for_each_candidate(a, S, xi, [&](uint32_t j, float4 xj) {
        float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
        if (s <= S.smax) {
            if (cnt < kMaxNb)
                lst[cnt++] = ((unsigned long long)(uint32_t)__float_as_int(xj.w) << 32) | j;
            else
                overflow = true;
        }
    });
    for (int q = 1; q < cnt; ++q) {
        unsigned long long v = lst[q];
        int r = q - 1;
        while (r >= 0 && lst[r] > v) {
            lst[r + 1] = lst[r];
            --r;
        }
        lst[r + 1] = v;
    }
    const float4* sp = a.spos + S.p_off;
    for (int q = 0; q < cnt; ++q) {
        uint32_t j = (uint32_t)(lst[q] & 0xffffffffu);
        f(j, __ldg(sp + j));
    }
    return !overflow;
}

// kernDefault for an in-range pair (fluid_system.h:410-416), times MASS.
__device__ __forceinline__ float density_term(const SceneDev& S, float len) {
    return fm(S.mass, fm(S.c_poly6, pow3(fs(S.hh, fm(len, len)))));
}

struct ForceAcc {
    float fpx, fpy, fpz;
    float fvx, fvy, fvz;
    float nx, ny, nz;
    float cfl;
    int nb;
    int any;
};

// Terms of passes 2 and 3 for one in-range pair (fluid_system.h:139-171):
// r = x_i - x_j, len = |r|; vj, Aj = P_j/rho_j^2, Bj = m/rho_j.
__device__ __forceinline__ void force_pair(const SceneDev& S, ForceAcc& acc, float rx, float ry, float rz,
                                           float len, float vix, float viy, float viz, float Ai, float4 vj,
                                           float Aj, float Bj, int idj, bool self) {
    // pass 3: colour-field Laplacian, self included (laplDefault, :424-428)
    {
        float ld = fm(fm(-S.c_grad, fs(S.hh, fm(len, len))),
                      fs(fm(fm(3.0f, S.h), S.h), fm(fm(7.0f, len), len)));
        acc.cfl = fa(acc.cfl, fm(Bj, ld));
    }
    if (self) return;
    acc.nb = max(acc.nb, idj);
    acc.any = 1;
    // gradPressure (:430-447)
    float gx, gy, gz;
    const float pw2 = pow2(fs(S.h, len));
    if (len < S.cthr) {
        float t = fm(fm(S.inv_sqrt3, S.c_spiky), pw2);
        gx = -t;
        gy = -t;
        gz = -t;
    } else {
        // glm::normalize: r * (1 / sqrt(dot(r, r))); the correctly rounded
        // reciprocal is the same value as the correctly rounded 1/len
        float inv = __frcp_rn(len);
        gx = -fm(fm(fm(rx, inv), S.c_spiky), pw2);
        gy = -fm(fm(fm(ry, inv), S.c_spiky), pw2);
        gz = -fm(fm(fm(rz, inv), S.c_spiky), pw2);
    }
    const float coef = fm(fa(Ai, Aj), S.mass);
    acc.fpx = fa(acc.fpx, fm(coef, gx));
    acc.fpy = fa(acc.fpy, fm(coef, gy));
    acc.fpz = fa(acc.fpz, fm(coef, gz));
    // laplVisc (:449-453)
    const float lv = fm(S.c_spiky, fs(S.h, len));
    acc.fvx = fa(acc.fvx, fm(fm(fs(vj.x, vix), Bj), lv));
    acc.fvy = fa(acc.fvy, fm(fm(fs(vj.y, viy), Bj), lv));
    acc.fvz = fa(acc.fvz, fm(fm(fs(vj.z, viz), Bj), lv));
    // gradDefault (:418-422)
    const float pw = pow2(fs(S.hh, fm(len, len)));
    acc.nx = fa(acc.nx, fm(Bj, -fm(fm(rx, S.c_grad), pw)));
    acc.ny = fa(acc.ny, fm(Bj, -fm(fm(ry, S.c_grad), pw)));
    acc.nz = fa(acc.nz, fm(Bj, -fm(fm(rz, S.c_grad), pw)));
}

// Fast-arithmetic form of density_term and force_pair (variant bit 17, fast
// mode only): the same kernel terms with the products grouped, fused
// multiply-adds, r^2 in place of |r|^2 and a hardware reciprocal square root
// for 1/|r|.  The in-range test stays exact (s <= smax), so the neighbour sets
// and NeighbId are the reference's; the rounding is not, and the results are
// held to the parity tolerance instead of to bits.
//
// r^2 with two fused multiply-adds, the force pass's fast form (its pairs
// are in range already): like dist2, within 3 units of rounding of the true
// sum of squares.
__device__ __forceinline__ float dist2_fma(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

__device__ __forceinline__ void force_pair_fast(const SceneDev& S, ForceAcc& acc, float rx, float ry, float rz,
                                                float s, float vix, float viy, float viz, float Ai, float4 vj,
                                                float Aj, float Bj, int idj, bool self) {
    const float hs = S.hh - s;  // h^2 - r^2
    // pass 3: colour-field Laplacian, self included (laplDefault)
    acc.cfl = fmaf(Bj, (-S.c_grad * hs) * fmaf(-7.0f, s, 3.0f * S.hh), acc.cfl);
    if (self) return;
    acc.nb = max(acc.nb, idj);
    acc.any = 1;
    const float coef = (Ai + Aj) * S.mass;
    if (s < S.cthr * S.cthr) {
        // coincident: gradPressure along normalize(1, 1, 1)
        const float hl = S.h - sqrtf(s);
        const float t = -(S.inv_sqrt3 * S.c_spiky) * (hl * hl);
        acc.fpx = fmaf(t, coef, acc.fpx);
        acc.fpy = fmaf(t, coef, acc.fpy);
        acc.fpz = fmaf(t, coef, acc.fpz);
        const float bl = Bj * (S.c_spiky * hl);
        acc.fvx = fmaf(vj.x - vix, bl, acc.fvx);
        acc.fvy = fmaf(vj.y - viy, bl, acc.fvy);
        acc.fvz = fmaf(vj.z - viz, bl, acc.fvz);
    } else {
        const float inv = rsqrtf(s);  // 1/|r|
        const float hl = fmaf(-s, inv, S.h);  // h - |r|
        const float g = -(S.c_spiky * coef) * (hl * hl) * inv;  // gradPressure / |r|, times coef
        acc.fpx = fmaf(rx, g, acc.fpx);
        acc.fpy = fmaf(ry, g, acc.fpy);
        acc.fpz = fmaf(rz, g, acc.fpz);
        const float bl = Bj * (S.c_spiky * hl);  // laplVisc times m/rho_j
        acc.fvx = fmaf(vj.x - vix, bl, acc.fvx);
        acc.fvy = fmaf(vj.y - viy, bl, acc.fvy);
        acc.fvz = fmaf(vj.z - viz, bl, acc.fvz);
    }
    const float gn = -(Bj * S.c_grad) * (hs * hs);  // gradDefault / r, times m/rho_j
    acc.nx = fmaf(rx, gn, acc.nx);
    acc.ny = fmaf(ry, gn, acc.ny);
    acc.nz = fmaf(rz, gn, acc.nz);
}

struct TSample {
    float y;
    float nx, ny, nz;
    int vnear;
};

// Heightfield surface at (x, z): bilinear over the vertex grid spanning the
// box floor (the repository's own contact model; the reference's
// Grid::collision is disabled at fluid_system.h:335-340).
__device__ __forceinline__ TSample terrain_at(const SceneDev& S, const float* hs, float x, float z) {
    TSample t;
    float fx = fm(fs(x, S.t_xlo), S.t_isx);
    float fz = fm(fs(z, S.t_zlo), S.t_isz);
    if (!(fx > 0.0f)) fx = 0.0f;
    if (fx > S.t_wmax) fx = S.t_wmax;
    if (!(fz > 0.0f)) fz = 0.0f;
    if (fz > S.t_dmax) fz = S.t_dmax;
    int i0 = (int)fx, j0 = (int)fz;
    if (i0 > S.tw - 2) i0 = S.tw - 2;
    if (j0 > S.td - 2) j0 = S.td - 2;
    const float tx = fs(fx, (float)i0), tz = fs(fz, (float)j0);
    const float* r0 = hs + S.t_off + (size_t)j0 * S.tw + i0;
    const float h00 = r0[0], h10 = r0[1];
    const float h01 = r0[S.tw], h11 = r0[S.tw + 1];
    const float a0 = fa(h00, fm(tx, fs(h10, h00)));
    const float a1 = fa(h01, fm(tx, fs(h11, h01)));
    const float hgt = fa(a0, fm(tz, fs(a1, a0)));
    t.y = fa(S.t_ylo, hgt);
    const float dx = fm(fa(fs(h10, h00), fm(tz, fs(fs(h11, h01), fs(h10, h00)))), S.t_isx);
    const float dz = fm(fs(a1, a0), S.t_isz);
    const float il = fdv(1.0f, fsq(fa(fa(fm(dx, dx), 1.0f), fm(dz, dz))));
    t.nx = fm(-dx, il);
    t.ny = il;
    t.nz = fm(-dz, il);
    int in = (int)fa(fx, 0.5f), jn = (int)fa(fz, 0.5f);
    if (in > S.tw - 1) in = S.tw - 1;
    if (jn > S.td - 1) jn = S.td - 1;
    t.vnear = jn * S.tw + in;
    return t;
}

// collisionS (fluid_system.h:355-407) for a box with centre c, half extents
// l and axis weights w (exactly 1 for the reference's cube).
__device__ __forceinline__ bool box_collide(const SceneDev& S, float px, float py, float pz, float* cp,
                                            float* nrm) {
    const float q[3] = {fs(px, S.box_c[0]), fs(py, S.box_c[1]), fs(pz, S.box_c[2])};
    const float aq[3] = {fabsf(q[0]), fabsf(q[1]), fabsf(q[2])};
    if (aq[0] < S.box_l[0] && aq[1] < S.box_l[1] && aq[2] < S.box_l[2]) return false;
    const float m0 = fm(aq[0], S.box_w[0]), m1 = fm(aq[1], S.box_w[1]), m2 = fm(aq[2], S.box_w[2]);
    int ax = 0;
    float maxp = m0;
    if (maxp < m1) {
        ax = 1;
        maxp = m1;
    }
    if (maxp < m2) ax = 2;
    cp[0] = px;
    cp[1] = py;
    cp[2] = pz;
    nrm[0] = nrm[1] = nrm[2] = 0.0f;
    float v, s;
    if (q[ax] < -S.box_l[ax]) {
        v = fs(S.box_c[ax], S.box_l[ax]);
        s = 1.0f;
    } else {
        v = fa(S.box_c[ax], S.box_l[ax]);
        s = -1.0f;
    }
    cp[ax] = v;
    nrm[ax] = s;
    return true;
}

__device__ __forceinline__ float len3(float x, float y, float z) { return fsq(dist2(x, y, z)); }

// ---------------------------------------------------------------------------
// Runs of equal values among the valid lanes of a warp (the valid lanes are a
// prefix, `mask`): the first lane of each run adds the run's length to
// counter[v] and every lane gets old value + its position in the run.  The
// state arrives in the previous step's sorted order, so particles of one cell
// are mostly adjacent and one atomic serves each cell.
struct Run {
    bool start;
    int leader;
    uint32_t len;
};

__device__ __forceinline__ Run run_of(uint32_t v, unsigned mask, int lane) {
    const uint32_t prev = __shfl_up_sync(mask, v, 1);
    Run r;
    r.start = lane == 0 || prev != v;
    const unsigned starts = __ballot_sync(mask, r.start);
    const unsigned upto = (2u << lane) - 1u;  // lanes 0..lane (all lanes for lane 31)
    r.leader = 31 - __clz(starts & upto);
    const unsigned above = starts & ~upto;
    const int end = above ? __ffs(above) - 1 : 32 - __clz(mask);
    r.len = (uint32_t)(end - lane);
    return r;
}

// keys: cell key of each particle, its slot within the cell (run-aggregated
// atomics) and the per-chunk totals that the scan needs.  The particles of a
// block are nearly all of one chunk, so the block adds that chunk's total once
// and only strays go to memory one by one: a system has a few hundred chunks, on
// a few dozen sectors, and an add per warp queued there (1,048,576 particles:
// 32,768 adds; keys of cells of h 33 -> 16 us, of h/2 29 -> 17; 8.4M rain 140 ->
// 81).  One tile a block: with the queue gone, four with their loads together
// are slower (20, 21, 90 us).
__global__ void __launch_bounds__(kMaxTile) k_keys(DevArrays a) {
    step_enter(a.early);
    __shared__ uint32_t s_chunk, s_sum;
    const int nwork = *a.n_ptiles;
    const int lane = threadIdx.x & 31;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        const int i = wk.start + threadIdx.x;
        const bool valid = i < S.p_off + S.n;
        const unsigned mask = __ballot_sync(kFull, valid);
        uint32_t k = 0, ck = 0;
        if (valid) {
            const float4 x = a.pos[i];
            const Cell c = cell_of(S, x.x, x.y, x.z);
            k = row_key(a.tab, S, c.cy, c.cz) + (uint32_t)c.cx;
            ck = k >> kChunkBits;
        }
        if (threadIdx.x == 0) {  // a tile's first particle is valid
            s_chunk = ck;
            s_sum = 0u;
        }
        __syncthreads();
        if (valid) {
            const Run r = run_of(k, mask, lane);
            uint32_t base = 0;
            if (r.start) base = atomicAdd(a.counts + S.k_off + k, r.len);
            const Run rc = run_of(ck, mask, lane);
            if (rc.start) {
                if (ck == s_chunk)
                    atomicAdd(&s_sum, rc.len);
                else
                    atomicAdd(a.chunk_sum + S.c_off + ck, rc.len);
            }
            a.key[i] = k;
            a.slot[i] = __shfl_sync(mask, base, r.leader) + (uint32_t)(lane - r.leader);
        }
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(a.chunk_sum + S.c_off + ck, s_sum);
    }
}

template <int NT>
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int q = 0; q < NT / 32; ++q) t += sh[q];
    return t;
}

template <int NT>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t u = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();
    if (lane == 31) sh[wid] = inc;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int q = 0; q < NT / 32; ++q)
        if (q < wid) before += sh[q];
    return before + inc - v;
}

// scan: exclusive prefix of the per-key counts within each scene, one chunk
// of kChunk keys per work item.  The chunk's offset is the sum of the earlier
// chunk totals of its scene, so no block waits on another.  Counts are
// cleared for the next step.
__global__ void __launch_bounds__(kScanThreads) k_scan(DevArrays a) {
    step_enter(a.early);
    __shared__ uint32_t sh[kScanThreads / 32];
    const int nwork = *a.n_ctiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ctiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        const int c = wk.start;
        uint32_t pre = 0;
        for (int j = threadIdx.x; j < c; j += kScanThreads) pre += a.chunk_sum[S.c_off + j];
        pre = block_sum<kScanThreads>(pre, sh);
        const size_t base = (size_t)S.k_off + (size_t)c * kChunk + (size_t)threadIdx.x * 16;
        uint4* cp = reinterpret_cast<uint4*>(a.counts + base);
        uint32_t v[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 t = cp[q];
            v[4 * q] = t.x;
            v[4 * q + 1] = t.y;
            v[4 * q + 2] = t.z;
            v[4 * q + 3] = t.w;
        }
        uint32_t run = 0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            uint32_t t = v[q];
            v[q] = run;
            run += t;
        }
        const uint32_t add = pre + block_exclusive<kScanThreads>(run, sh);
        uint4* op = reinterpret_cast<uint4*>(a.offsets + base);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            op[q] = make_uint4(v[4 * q] + add, v[4 * q + 1] + add, v[4 * q + 2] + add, v[4 * q + 3] + add);
            cp[q] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
    }
}

// scatter: place each particle's index at its cell's offset + slot, and clear
// the chunk totals (the scan that read them has finished).
__global__ void __launch_bounds__(kMaxTile) k_scatter(DevArrays a) {
    step_enter(a.early);
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        const int i = wk.start + threadIdx.x;
        if (i < S.p_off + S.n) {
            const uint32_t dst = a.offsets[S.k_off + a.key[i]] + a.slot[i];
            if (dst < (uint32_t)S.n)
                a.perm[S.p_off + dst] = (uint32_t)i;
            else
                atomicOr(a.status, 2u);  // inconsistent counts: never write out of range
        }
        const int t = (wk.start - S.p_off) / (int)blockDim.x;
        const int ntiles = (S.n + (int)blockDim.x - 1) / (int)blockDim.x;
        for (int j = t * (int)blockDim.x + (int)threadIdx.x; j < S.nchunks; j += ntiles * (int)blockDim.x)
            a.chunk_sum[S.c_off + j] = 0u;
    }
}

// reorder: make the order within each cell stable (ascending previous index,
// so results never depend on atomic arrival order) and gather the state into
// the sorted arrays.
__global__ void __launch_bounds__(kMaxTile) k_reorder(DevArrays a) {
    step_enter(a.early);
    const int nwork = *a.n_ptiles;
    if (a.ctr && blockIdx.x == 0 && threadIdx.x < 2) a.ctr[threadIdx.x] = 0u;  // for this step's neighbour kernels
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        const int p = wk.start + threadIdx.x;
        if (p >= S.p_off + S.n) continue;
        const uint32_t i = a.perm[p];
        if (i < (uint32_t)S.p_off || i >= (uint32_t)(S.p_off + S.n)) {
            atomicOr(a.status, 2u);
            continue;
        }
        const uint32_t k = a.key[i];
        const uint32_t st = a.offsets[S.k_off + k];
        const uint32_t en = min(a.offsets[S.k_off + k + 1], (uint32_t)S.n);
        const uint32_t* cell = a.perm + S.p_off;
        uint32_t r = 0;
        for (uint32_t q = st; q < en; ++q) r += (cell[q] < i) ? 1u : 0u;
        if (st + r >= (uint32_t)S.n) {
            atomicOr(a.status, 2u);
            continue;
        }
        const int dst = S.p_off + (int)(st + r);
        a.spos[dst] = a.pos[i];
        a.svel[dst] = a.vel[i];
        if (S.flags & kFlagRecord) a.snbid[dst] = a.nbid[i];
    }
}

// The whole sort of a small scene in one block: keys, scan, scatter and reorder
// with the counts, offsets and order in shared memory.  The four kernels are
// chains of dependent loads of 5 to 9 us each at these sizes, whatever the
// number of particles.  The work list of a system that takes this sort begins with
// the scenes' first tiles: block w takes the scene of item w.
constexpr int kSortThreads = 1024;
constexpr int kSortPer = kSmallSort / kSortThreads;  // particles a thread takes

__global__ void __launch_bounds__(kSortThreads) k_sort_small(const __grid_constant__ DevArrays a) {
    step_enter(a.early);
    extern __shared__ uint32_t sm[];
    __shared__ uint32_t s_warp[kSortThreads / 32];
    const int tid = threadIdx.x;
    if (a.ctr && blockIdx.x == 0 && tid < 2) a.ctr[tid] = 0u;  // for this step's neighbour kernels
    const Work wk = a.ptiles[blockIdx.x];
    const SceneDev& S = a.scenes[wk.scene];
    if (a.steps_left[wk.scene] == 0) return;
    const int n = S.n, nkeys = S.nkeys;
    const int per = ((nkeys + kSortThreads - 1) / kSortThreads) | 1;  // keys a thread scans; odd: no bank conflicts
    uint32_t* perm = sm;                 // kSmallSort
    uint32_t* cnt = sm + kSmallSort;     // per * kSortThreads: counts, then offsets
    float4 x[kSortPer], v[kSortPer];
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
        const int i = tid + u * kSortThreads;
        if (i < n) x[u] = a.pos[S.p_off + i], v[u] = a.vel[S.p_off + i];
    }
    for (int k = tid; k < per * kSortThreads; k += kSortThreads) cnt[k] = 0u;
    __syncthreads();
    uint32_t key[kSortPer], slot[kSortPer];
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
        const int i = tid + u * kSortThreads;
        if (i >= n) continue;
        const Cell c = cell_of(S, x[u].x, x[u].y, x[u].z);
        key[u] = row_key(a.tab, S, c.cy, c.cz) + (uint32_t)c.cx;
        a.key[S.p_off + i] = key[u];
        slot[u] = atomicAdd(cnt + key[u], 1u);
    }
    __syncthreads();
    uint32_t sum = 0;
    for (int k = 0; k < per; ++k) sum += cnt[tid * per + k];
    uint32_t run = block_exclusive<kSortThreads>(sum, s_warp);
    for (int k = 0; k < per; ++k) {
        const uint32_t c = cnt[tid * per + k];
        cnt[tid * per + k] = run;
        run += c;
    }
    __syncthreads();
    for (int k = tid; k < nkeys; k += kSortThreads) a.offsets[S.k_off + k] = cnt[k];
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
        const int i = tid + u * kSortThreads;
        if (i < n) perm[cnt[key[u]] + slot[u]] = (uint32_t)i;
    }
    __syncthreads();
    // stable within each cell: the rank by previous index
#pragma unroll
    for (int u = 0; u < kSortPer; ++u) {
        const int i = tid + u * kSortThreads;
        if (i >= n) continue;
        const uint32_t st = cnt[key[u]], en = cnt[key[u] + 1];
        uint32_t r = st;
        for (uint32_t q = st; q < en; ++q) r += perm[q] < (uint32_t)i ? 1u : 0u;
        const int dst = S.p_off + (int)r;
        a.spos[dst] = x[u];
        a.svel[dst] = v[u];
        if (S.flags & kFlagRecord) a.snbid[dst] = a.nbid[S.p_off + i];
    }
}

// Where entry q of the neighbour list of lane l of a tile of T particles is,
// from the tile's start: groups of four entries, the lanes' groups side by
// side.
__device__ __forceinline__ uint32_t list_at(int q, int l, int T) {
    return ((uint32_t)(q >> 2) * (uint32_t)T + (uint32_t)l) * 4u + (uint32_t)(q & 3);
}

// Work slices of the neighbour kernels.  Static: block b takes the tiles b,
// b + gridDim.x, ..., and its thread t the tile's lane t.  Dynamic (DYN):
// every warp takes the next 32-lane slice of any tile from a counter, so no
// warp slot waits for the slowest warp of its block.  Which warp computes a
// particle changes nothing in what it computes.
template <bool DYN>
__device__ __forceinline__ int next_slice(unsigned* ctr, int cur) {
    if (!DYN) return cur + (int)gridDim.x;
    int t = 0;
    if ((threadIdx.x & 31) == 0) t = (int)atomicAdd(ctr, 1u);
    return __shfl_sync(kFull, t, 0);
}

template <bool DYN>
__device__ __forceinline__ int first_slice(unsigned* ctr) {
    return DYN ? next_slice<true>(ctr, 0) : (int)blockIdx.x;
}

// density: pass 1 (fluid_system.h:107-124), then the per-particle factors the
// force pass reuses: P/rho^2 and m/rho.
// LISTED: the in-range pairs are compacted (for_each_in_range_listed) instead
// of evaluated inside the candidate loop; which one is faster depends on the
// neighbour density, so the autotuner picks it.
template <bool ORDERED, bool LISTED, int MINB>
__global__ void __launch_bounds__(kMaxTile, MINB) k_density(DevArrays a) {
    extern __shared__ uint32_t list[];
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if (((S.flags & kFlagOrdered) != 0) != ORDERED) continue;
        const int p = wk.start + (int)threadIdx.x;
        const bool valid = p < S.p_off + S.n;
        if ((ORDERED || !LISTED) && !valid) continue;
        const float4 xi = a.spos[valid ? p : S.p_off];
        float rho = 0.0f;
        if (ORDERED) {
            auto term = [&](uint32_t, float4 xj) {
                float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                if (s <= S.smax) rho = fa(rho, density_term(S, fsq(s)));
            };
            if (!for_each_in_range_ordered(a, S, xi, term)) atomicOr(a.status, 1u);
        } else if (LISTED) {
            const float4* sp = a.spos + S.p_off;
            for_each_in_range_listed(a, S, valid, xi, list, [&](uint32_t j) {
                const float4 xj = __ldg(sp + j);
                const float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                rho = fa(rho, density_term(S, fsq(s)));
            });
            if (!valid) continue;
        } else {
            for_each_candidate(a, S, xi, [&](uint32_t, float4 xj) {
                const float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                if (s <= S.smax) rho = fa(rho, density_term(S, fsq(s)));
            });
        }
        const float P = fm(S.k, fs(rho, S.p0));
        const float Ai = fdv(P, fm(rho, rho)), Bi = fdv(S.mass, rho);
        a.dyn[p] = make_float4(rho, Ai, Bi, P);
    }
}

// dist2 of two candidates from the particle at (-nx, -ny, -nz), both at once.
__device__ __forceinline__ f2 dist2_two(float4 x0, float4 x1, float nx, float ny, float nz, f2 nzero) {
    const f2 dx = pk(fa(x0.x, nx), fa(x1.x, nx)), dy = pk(fa(x0.y, ny), fa(x1.y, ny)),
             dz = pk(fa(x0.z, nz), fa(x1.z, nz));
    return add2(add2(mulr2(dx, dx, nzero), mulr2(dy, dy, nzero)), mulr2(dz, dz, nzero));
}

// for_rows_r with its loads ahead of their use: while one row's candidates are
// visited, the next row's two offsets and the row number of the one after are
// on their way.
template <int R, class Fn>
__device__ __forceinline__ void for_rows_ahead(const DevArrays& a, const SceneDev& S, float4 xi, bool valid, Fn&& fn) {
    const Probe q = probe_of(S, xi);
    const uint32_t* off = a.offsets + S.k_off + q.c.cx;
    const float H2 = S.hcell * S.hcell;
    constexpr int XS = R == 1 ? 2 : 1, RX = R * XS, side = 2 * R + 1;
    float gx2[2 * RX + 1];
#pragma unroll
    for (int d = -RX; d <= RX; ++d) {
        const int k = q.c.cx + d;
        float g2 = INFINITY;
        if (k >= 0 && k < S.nx) {
            const float g = cell_gap(q.tx, k, S.nx) * (1.0f / XS);
            g2 = g * g;
        }
        gx2[d + RX] = g2;
    }
    const int nx = S.nx, ny = S.ny, nz = S.nz;
    const uint32_t* tab = a.tab + S.tab_off;
    int y = q.c.cy - R, z = q.c.cz - R;
    float z2 = INFINITY;  // squared gap of slab z
    auto slab = [&]() {
        z2 = INFINITY;
        if (valid && q.finite && z >= 0 && z < nz) {
            const float g = cell_gap(q.tz, z, nz);
            z2 = g * g;
        }
    };
    slab();
    uint32_t num = 0, st = 0, en = 0;  // row number; next range
    int lohi = -1;                     // its cells (-1: not reached)
#pragma unroll 1
    for (int r = 0; r < side * side + 2; ++r) {
        const uint32_t cst = st, cen = en;
        st = en = 0;
        if (lohi >= 0) {
            const uint32_t* o = off + num * (uint32_t)nx;
            st = __ldg(o - (lohi >> 4));
            en = __ldg(o + (lohi & 15) + 1);
        }
        lohi = -1;
        if (r < side * side) {
            if (y >= 0 && y < ny) {
                const float g = cell_gap(q.ty, y, ny);
                const float r2 = H2 - g * g - z2;
                if (r2 >= 0.0f) {
                    int l = 0, h = 0;
#pragma unroll
                    for (int d = 1; d <= RX; ++d) {
                        if (gx2[RX - d] <= r2) l = d;
                        if (gx2[RX + d] <= r2) h = d;
                    }
                    lohi = l * 16 + h;
                    num = __ldg(tab + z * ny + y);
                }
            }
            if (++y > q.c.cy + R) {
                y = q.c.cy - R;
                ++z;
                slab();
            }
        }
        fn(cst, cen);
    }
}

// Entries of a lane's buffer (ListOut), which is emptied, and read to its end, in
// groups of four.
constexpr int kBuf = 28;
static_assert(kBuf % 4 == 0 && kBuf >= 8, "whole groups, and room for four beside one");

// One lane's neighbour list while it is written.  The lanes of a warp are at
// different entries, so an index stored by itself is four bytes to a sector of
// its own: 61 million sectors a launch at 1,048,576 particles and cells of h,
// half of the L1-to-L2 path's time, and L2 wrote some of them out half filled
// (DRAM 406 MB written for 280).  Here the indices go to the lane's column of
// a buffer in shared memory and from there to the list in groups of four, all
// lanes together: 3,291 -> 2,672 us for the 8.4M rain in fast arithmetic.  28
// entries a lane: 16 empty it too often (2,824), 24 take 2,703; the buffer is
// sized by the tile, since what it takes is lost to the candidates' L1.
struct ListOut {
    uint32_t* nl;      // the lane's group 0
    uint32_t stride;   // words from one of its groups to the next
    uint32_t* col;     // the lane's column
    uint32_t* next;    // its first free entry
    int flushed;

    __device__ __forceinline__ int pending() const { return (int)(next - col) >> 5; }
    __device__ __forceinline__ void add(uint32_t j) {
        *next = j;
        next += 32;
    }
    __device__ __forceinline__ void flush() {
        int n = pending();
        uint32_t* from = col;
        for (; n >= 4; n -= 4, from += 128) {
            const uint32_t e0 = from[0], e1 = from[32], e2 = from[64], e3 = from[96];
            if (flushed < kNbCap) {
                *reinterpret_cast<uint4*>(nl + (size_t)((uint32_t)(flushed >> 2) * stride)) = make_uint4(e0, e1, e2, e3);
            }
            flushed += 4;
        }
        if (from != col) {
            if (n > 0) col[0] = from[0];
            if (n > 1) col[32] = from[32];
            if (n > 2) col[64] = from[64];
            next = col + 32 * n;
        }
    }
    __device__ __forceinline__ void make_room() {  // for four more in every lane
        if (__any_sync(kFull, next > col + 32 * (kBuf - 4))) flush();
    }
    __device__ __forceinline__ int finish() {
        const int cnt = flushed + pending();
        while (flushed < cnt) {  // the last group may hold entries past the end
            if (flushed < kNbCap)
                *reinterpret_cast<uint4*>(nl + (size_t)((uint32_t)(flushed >> 2) * stride)) =
                    make_uint4(col[0], col[32], col[64], col[96]);
            flushed += 4;
            col += 128;
        }
        return cnt;
    }
};

// Tests the candidates [st, en) of a row, each lane its own, four at a time in
// straight-line code: packed differences and squares, a compare each,
// predicated appends of the in-range indices; with fast arithmetic also the
// density term.  All lanes of the warp take part, for its longest row.
template <bool FM>
__device__ __forceinline__ void density_row(const SceneDev& S, const float4* sp, float nx, float ny, float nz, f2 nzero,
                                            uint32_t st, uint32_t en, ListOut& out, float& rho) {
    const float smax = S.smax, hh = S.hh, mc = S.mass * S.c_poly6;
    auto hit = [&](bool in, uint32_t j, float c3) {
        if (in) {
            if (FM) rho = fmaf(mc, c3, rho);
            out.add(j);
        }
    };
    const int longest = __reduce_max_sync(kFull, (int)(en - st));
    for (int t = 0; t < longest; t += 4) {
        out.make_room();
        const uint32_t j = st + t;
        const bool m0 = j < en, m1 = j + 1 < en, m2 = j + 2 < en, m3 = j + 3 < en;
        const float4* c = sp + j;
        float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0, x2 = x0, x3 = x0;
        if (m0) x0 = __ldg(c);
        if (m1) x1 = __ldg(c + 1);
        if (m2) x2 = __ldg(c + 2);
        if (m3) x3 = __ldg(c + 3);
        const f2 sa = dist2_two(x0, x1, nx, ny, nz, nzero), sb = dist2_two(x2, x3, nx, ny, nz, nzero);
        f2 ca = 0, cb = 0;
        if (FM) {
            const f2 ha = fma2(sa, pk(-1.0f), pk(hh)), hb = fma2(sb, pk(-1.0f), pk(hh));
            ca = mul2(mul2(ha, ha), ha);
            cb = mul2(mul2(hb, hb), hb);
        }
        hit(m0 && lo(sa) <= smax, j, lo(ca));
        hit(m1 && hi(sa) <= smax, j + 1, hi(ca));
        hit(m2 && lo(sb) <= smax, j + 2, lo(cb));
        hit(m3 && hi(sb) <= smax, j + 3, hi(cb));
    }
}

// Sum of the exact density terms over a finished list, four entries at a time
// with the next four loaded ahead; the cells again when the list overflowed.
__device__ __forceinline__ float density_sum_exact(const DevArrays& a, const SceneDev& S, float4 xi, const uint32_t* nl,
                                                   uint32_t stride, int cnt, f2 nzero) {
    const float4* sp = a.spos + S.p_off;
    float rho = 0.0f;
    if (cnt > kNbCap) {
        for_each_candidate(a, S, xi, [&](uint32_t, float4 xj) {
            const float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
            if (s <= S.smax) rho = fa(rho, density_term(S, fsq(s)));
        });
        return rho;
    }
    const float nx = -xi.x, ny = -xi.y, nz = -xi.z;
    uint4 e = make_uint4(0, 0, 0, 0);
    if (0 < cnt) e = *reinterpret_cast<const uint4*>(nl);
    for (int q = 0; q < cnt; q += 4) {
        nl += stride;
        const uint32_t j[4] = {e.x, q + 1 < cnt ? e.y : e.x, q + 2 < cnt ? e.z : e.x, q + 3 < cnt ? e.w : e.x};
        float4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = __ldg(sp + j[u]);
        if (q + 4 < cnt) e = *reinterpret_cast<const uint4*>(nl);
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            const f2 s2 = dist2_two(x[u], x[u + 1], nx, ny, nz, nzero);
            const f2 l2 = pk(fsq(lo(s2)), fsq(hi(s2)));
            // mass * (c * pow3(hh - len * len)), pow3 as above
            const f2 v = fma2(mulr2(l2, l2, nzero), pk(-1.0f), pk(S.hh));
            const f2 pp = mul2(v, v), w = fma2(v, v, mul2(pp, pk(-1.0f)));
            const f2 c = mulr2(pp, v, nzero), f = fma2(pp, v, mul2(c, pk(-1.0f)));
            const f2 t = mulr2(pk(S.mass), mul2(pk(S.c_poly6), add2(c, fma2(w, v, f))), nzero);
            if (q + u < cnt) rho = fa(rho, lo(t));
            if (q + u + 1 < cnt) rho = fa(rho, hi(t));
        }
    }
    return rho;
}

// density with the neighbour lists (variant bit 3), one lane per particle.  The
// fast arithmetic adds its short term in place; the exact form, whose term has
// a square root, sums over the finished list, where every lane of the warp has
// a pair to evaluate.  No unit bounds it (instructions 65%, L1 data path 60%):
// the rows are walked in step, which keeps a warp's loads in few cache lines
// but leaves 40% of the lanes waiting for the longest row.  80 registers: with 64
// or 72 the loads of four candidates are no longer all in flight (exact, cells
// of h: 535 and 478 us where these take 435; fast, cells of h/2: 409 and 351,
// 312), and 16 warps an SM are too few (392).  1,048,576 particles, before and after: fast, cells of h/2, 380 ->
// 315 us; exact, cells of h, 488 -> 439 us.
template <bool FM>
__global__ void __launch_bounds__(kMaxTile, 3) k_density_list(const __grid_constant__ DevArrays a, bool pack) {
    extern __shared__ uint32_t buf[];  // kBuf x 32 words a warp
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev S = a.scenes[wk.scene];  // by value: the list stores cannot alias it
        if ((S.flags & kFlagOrdered) != 0) continue;
        const int p = wk.start + (int)threadIdx.x;
        const bool valid = p < S.p_off + S.n;
        const float4 xi = a.spos[valid ? p : S.p_off];
        const float4* sp = a.spos + S.p_off;
        uint32_t* col = buf + (threadIdx.x >> 5) * (kBuf * 32) + (threadIdx.x & 31);
        ListOut out = {a.nlist + (size_t)wk.start * kNbCap + 4 * threadIdx.x, 4 * blockDim.x, col, col, 0};
        float rho = 0.0f;
        const f2 nzero = neg_zero();
        auto row = [&](uint32_t st, uint32_t en) {
            density_row<FM>(S, sp, -xi.x, -xi.y, -xi.z, nzero, st, en, out, rho);
        };
        if (S.reach == 1)
            for_rows_ahead<1>(a, S, xi, valid, row);
        else if (S.reach == 2)
            for_rows_ahead<2>(a, S, xi, valid, row);
        else
            for_rows_any(a, S, xi, valid, row);
        const int cnt = out.finish();
        if (!valid) continue;
        if (!FM) rho = density_sum_exact(a, S, xi, out.nl, out.stride, cnt, nzero);
        a.ncnt[p] = cnt;
        const float P = fm(S.k, fs(rho, S.p0));
        const float Ai = fdv(P, fm(rho, rho)), Bi = fdv(S.mass, rho);
        a.dyn[p] = make_float4(rho, Ai, Bi, P);
        if (pack) {
            const float4 vi = a.svel[p];
            a.fdat[2 * (size_t)p] = make_float4(xi.x, xi.y, xi.z, Ai);
            a.fdat[2 * (size_t)p + 1] = make_float4(vi.x, vi.y, vi.z, Bi);
        }
    }
}

// Pass-2 results (fluid_system.h:151-154), pass 3 (:163, :177) and advance
// (:306-353) with the terrain contact, the box collision and the erosion
// exchange, from a particle's neighbour sums; only a writer stores the state
// and the record and adds the exchange to the terrain.
__device__ __forceinline__ void integrate_and_store(const DevArrays& a, const SceneDev& S, int p, float4 xi, float4 vi,
                                                    float rho, const ForceAcc& acc, bool writer) {
    // pass-2 results (:151-154) and pass 3 (:163, :177)
    const float Fpx = -fm(acc.fpx, rho), Fpy = -fm(acc.fpy, rho), Fpz = -fm(acc.fpz, rho);
    const float Fvx = fm(acc.fvx, S.visc), Fvy = fm(acc.fvy, S.visc), Fvz = fm(acc.fvz, S.visc);
    const float Fgx = fm(rho, S.g[0]), Fgy = fm(rho, S.g[1]), Fgz = fm(rho, S.g[2]);
    const float nsig = fm(-S.sigma, acc.cfl);
    const float Fsx = fm(nsig, acc.nx), Fsy = fm(nsig, acc.ny), Fsz = fm(nsig, acc.nz);
    // advance (:318-331)
    const float Fx = fa(fa(Fpx, Fvx), fa(Fgx, Fsx));
    const float Fy = fa(fa(Fpy, Fvy), fa(Fgy, Fsy));
    const float Fz = fa(fa(Fpz, Fvz), fa(Fgz, Fsz));
    const float ax = fdv(Fx, rho), ay = fdv(Fy, rho), az = fdv(Fz, rho);
    const float dt = S.dt;
    float vx = fa(vi.x, fm(ax, dt)), vy = fa(vi.y, fm(ay, dt)), vz = fa(vi.z, fm(az, dt));
    float px = fa(xi.x, fm(vx, dt)), py = fa(xi.y, fm(vy, dt)), pz = fa(xi.z, fm(vz, dt));

    const bool has_t = (S.flags & kFlagTerrain) != 0;
    TSample ts;
    if (has_t) {
        ts = terrain_at(S, a.theight, px, pz);
        if (py < ts.y && dt != 0.0f) {
            const float d = fs(ts.y, py);
            const float vdn = fa(fa(fm(vx, ts.nx), fm(vy, ts.ny)), fm(vz, ts.nz));
            if (vdn < 0.0f) {
                const float sp = len3(vx, vy, vz);
                const float f = fa(1.0f, sp > 0.0f ? fdv(fm(S.cr, d), fm(dt, sp)) : 0.0f);
                vx = fs(vx, fm(fm(ts.nx, f), vdn));
                vy = fs(vy, fm(fm(ts.ny, f), vdn));
                vz = fs(vz, fm(fm(ts.nz, f), vdn));
            }
            py = ts.y;
        }
    }
    bool moved = false;
    {
        float cp[3], nr[3];
        if (box_collide(S, px, py, pz, cp, nr) && dt != 0.0f) {
            const float d = len3(fs(px, cp[0]), fs(py, cp[1]), fs(pz, cp[2]));
            const float f = fa(1.0f, fdv(fm(0.5f, d), fm(dt, len3(vx, vy, vz))));
            const float vdn = fa(fa(fm(vx, nr[0]), fm(vy, nr[1])), fm(vz, nr[2]));
            vx = fs(vx, fm(fm(nr[0], f), vdn));
            vy = fs(vy, fm(fm(nr[1], f), vdn));
            vz = fs(vz, fm(fm(nr[2], f), vdn));
            moved = px != cp[0] || pz != cp[2];
            px = cp[0];
            py = cp[1];
            pz = cp[2];
        }
    }
    int sed = __float_as_int(vi.w);
    if (has_t && (S.flags & kFlagErosion)) {
        // the exchange uses the surface under the particle's final
        // position: a wall that moved it in x or z moved it to another
        // sample of the terrain
        if (moved) ts = terrain_at(S, a.theight, px, pz);
        const float e = fs(py, ts.y);
        if (e <= S.layer) {
            float capf = fm(S.k_capacity, len3(vx, vy, vz));
            if (capf > 1.0f) capf = 1.0f;
            const float cap = fm(capf, 1073741824.0f);
            const float s = __int2float_rn(sed);
            const float q = (s < cap) ? fm(fm(S.k_pick, dt), fs(cap, s)) : -fm(fm(S.k_dep, dt), fs(s, cap));
            if (q == q) {
                long long Q = __float2ll_rn(q);
                if ((long long)sed + Q < 0) Q = -(long long)sed;
                if ((long long)sed + Q > 1073741824LL) Q = 1073741824LL - (long long)sed;
                if (Q != 0) {
                    sed += (int)Q;
                    if (writer)
                        atomicAdd(reinterpret_cast<unsigned long long*>(a.tdelta + S.t_off + ts.vnear),
                                  (unsigned long long)(-Q));
                }
            }
        }
    }
    if (!writer) return;
    a.pos[p] = make_float4(px, py, pz, xi.w);
    a.vel[p] = make_float4(vx, vy, vz, __int_as_float(sed));
    if (S.flags & kFlagRecord) {
        float* r = a.rec + (size_t)p * kRecFloats;
        r[0] = ax; r[1] = ay; r[2] = az;
        r[3] = Fpx; r[4] = Fpy; r[5] = Fpz;
        r[6] = Fvx; r[7] = Fvy; r[8] = Fvz;
        r[9] = Fgx; r[10] = Fgy; r[11] = Fgz;
        r[12] = Fsx; r[13] = Fsy; r[14] = Fsz;
        r[15] = acc.nx; r[16] = acc.ny; r[17] = acc.nz;
        a.nbid[p] = acc.any ? acc.nb : a.snbid[p];
    }
}

// force: passes 2 and 3 (fluid_system.h:127-178) and advance (:306-353) with
// the terrain contact, the box collision and the erosion exchange.
// NL: the in-range neighbours come from the lists the density pass wrote
// (same order as the traversal, so the same sums), list entries two ahead and
// the neighbour's state one ahead; a particle whose list overflowed walks its
// cells instead.  This form gathers from the three sorted arrays: it serves
// systems whose HBM budget has no room for the packed records (k_force_rec).
template <bool ORDERED, int MINB, bool NL = false, bool DYN = false, bool FM = false>
__global__ void __launch_bounds__(kMaxTile, MINB) k_force(DevArrays a) {
    extern __shared__ uint32_t list[];
    const int nwork = *a.n_ptiles;
    const int spt = DYN ? a.tile / 32 : 1;  // slices per tile
    for (int sl = first_slice<DYN>(a.ctr + 1); sl < nwork * spt; sl = next_slice<DYN>(a.ctr + 1, sl)) {
        const int w = DYN ? sl / spt : sl;
        const int li = DYN ? (sl % spt) * 32 + (int)(threadIdx.x & 31) : (int)threadIdx.x;  // lane within the tile
        const int lstride = DYN ? a.tile : (int)blockDim.x;
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if (((S.flags & kFlagOrdered) != 0) != ORDERED) continue;
        const int p0 = wk.start + li;
        const bool valid = p0 < S.p_off + S.n;
        if (ORDERED && !valid) continue;
        const int p = valid ? p0 : S.p_off;
        const int pl = p - S.p_off;
        const float4 xi = a.spos[p];
        const float4 vi = a.svel[p];
        const float4 di = a.dyn[p];
        const float rho = di.x, Ai = di.y;
        ForceAcc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
        const float4* sp = a.spos + S.p_off;
        const float4* sv = a.svel + S.p_off;
        const float4* sd = a.dyn + S.p_off;
        auto pair_with = [&](uint32_t j, float4 xj, float4 vj, float4 dj) {
            const float rx = fs(xi.x, xj.x), ry = fs(xi.y, xj.y), rz = fs(xi.z, xj.z);
            const float s = FM ? dist2_fma(rx, ry, rz) : dist2(rx, ry, rz);
            if (FM)
                force_pair_fast(S, acc, rx, ry, rz, s, vi.x, vi.y, vi.z, Ai, vj, dj.y, dj.z, __float_as_int(xj.w),
                                (int)j == pl);
            else
                force_pair(S, acc, rx, ry, rz, fsq(s), vi.x, vi.y, vi.z, Ai, vj, dj.y, dj.z, __float_as_int(xj.w),
                           (int)j == pl);
        };
        auto pair = [&](uint32_t j, float4 xj) { pair_with(j, xj, __ldg(sv + j), __ldg(sd + j)); };
        if (ORDERED) {
            // the ordered list holds only in-range candidates
            if (!for_each_in_range_ordered(a, S, xi, pair)) atomicOr(a.status, 1u);
        } else {
            const int cnt = (NL && valid) ? a.ncnt[p] : 0;
            if (!NL) {
                for_each_in_range_listed(a, S, valid, xi, list, [&](uint32_t j) { pair(j, __ldg(sp + j)); });
            } else if (cnt > kNbCap) {
                // the list overflowed: this lane walks its cells (same order)
                for_each_candidate(a, S, xi, [&](uint32_t j, float4 xj) {
                    if (dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z)) <= S.smax) pair(j, xj);
                });
            } else {
                const uint32_t* nl = a.nlist + (size_t)wk.start * kNbCap;
                auto entry = [&](int q) { return q < cnt ? __ldg(nl + list_at(q, li, lstride)) : 0u; };
                uint32_t j0 = entry(0), j1 = entry(1);
                float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), v0 = x0, d0 = x0;
                if (cnt > 0) {
                    x0 = __ldg(sp + j0);
                    v0 = __ldg(sv + j0);
                    d0 = __ldg(sd + j0);
                }
                for (int q = 0; q < cnt; ++q) {
                    const uint32_t j2 = entry(q + 2);
                    float4 x1 = x0, v1 = v0, d1 = d0;
                    if (q + 1 < cnt) {
                        x1 = __ldg(sp + j1);
                        v1 = __ldg(sv + j1);
                        d1 = __ldg(sd + j1);
                    }
                    pair_with(j0, x0, v0, d0);
                    j0 = j1;
                    j1 = j2;
                    x0 = x1;
                    v0 = v1;
                    d0 = d1;
                }
            }
            if (!valid) continue;
        }
        integrate_and_store(a, S, p, xi, vi, rho, acc, true);
    }
}

// Sum of the pair terms of two list neighbours A and B (A first), the terms
// of both computed together in packed operations; each term and each sum
// rounds as in force_pair (FM: force_pair_fast).  nr = x_j - x_i is the
// negative of the reference's r and every coefficient that multiplies it is
// negated, which changes no bits.  The particle itself (s = 0) needs no test:
// its r and its velocity difference are zero, so it adds zeros to all sums but
// the colour field's, where it belongs; only the reciprocal length is kept
// finite.  Coincident neighbours (s below the threshold) must not come here.
struct PairIn {
    float x, y, z;     // x_j - x_i
    float vx, vy, vz;  // v_j - v_i
    float AA, B;       // A_i + A_j, m/rho_j
    float s;           // |x_j - x_i|^2
};

struct PairConst {
    float h, hh, hh3, cg, cs, mass, clamp;
    f2 nzero;
};

template <bool FM>
__device__ __forceinline__ void force_two(const PairConst& K, ForceAcc& acc, const PairIn& a, const PairIn& b,
                                          float lapB) {
    const f2 S2 = pk(a.s, b.s);
    if (FM) {
        const f2 hs = fma2(S2, pk(-1.0f), pk(K.hh));
        const f2 lap = mul2(mul2(hs, pk(K.cg)), fma2(S2, pk(-7.0f), pk(K.hh3)));
        acc.cfl = fmaf(-a.B, lo(lap), acc.cfl);
        acc.cfl = fmaf(-lapB, hi(lap), acc.cfl);
        const f2 inv = pk(rsqrtf(fmaxf(a.s, K.clamp)), rsqrtf(fmaxf(b.s, K.clamp)));
        const f2 w = fma2(S2, inv, pk(-K.h));  // |r| - h
        const f2 coef = mul2(pk(a.AA, b.AA), pk(K.mass));
        const f2 g = mul2(mul2(mul2(coef, pk(K.cs)), mul2(w, w)), inv);
        const f2 lv = mul2(w, pk(K.cs));
        const f2 gn = mul2(mul2(pk(a.B, b.B), pk(K.cg)), mul2(hs, hs));
        const f2 bl = mul2(pk(a.B, b.B), lv);
        acc.fpx = fmaf(a.x, lo(g), acc.fpx);
        acc.fpy = fmaf(a.y, lo(g), acc.fpy);
        acc.fpz = fmaf(a.z, lo(g), acc.fpz);
        acc.fvx = fmaf(a.vx, -lo(bl), acc.fvx);
        acc.fvy = fmaf(a.vy, -lo(bl), acc.fvy);
        acc.fvz = fmaf(a.vz, -lo(bl), acc.fvz);
        acc.nx = fmaf(a.x, lo(gn), acc.nx);
        acc.ny = fmaf(a.y, lo(gn), acc.ny);
        acc.nz = fmaf(a.z, lo(gn), acc.nz);
        acc.fpx = fmaf(b.x, hi(g), acc.fpx);
        acc.fpy = fmaf(b.y, hi(g), acc.fpy);
        acc.fpz = fmaf(b.z, hi(g), acc.fpz);
        acc.fvx = fmaf(b.vx, -hi(bl), acc.fvx);
        acc.fvy = fmaf(b.vy, -hi(bl), acc.fvy);
        acc.fvz = fmaf(b.vz, -hi(bl), acc.fvz);
        acc.nx = fmaf(b.x, hi(gn), acc.nx);
        acc.ny = fmaf(b.y, hi(gn), acc.ny);
        acc.nz = fmaf(b.z, hi(gn), acc.nz);
    } else {
        const float la = fsq(a.s), lb = fsq(b.s);
        const f2 cg = pk(K.cg);
        const f2 L = pk(la, lb);
        const f2 hs = fma2(mulr2(L, L, K.nzero), pk(-1.0f), pk(K.hh));
        const f2 lap = mul2(mul2(cg, hs), fma2(mulr2(mul2(pk(7.0f), L), L, K.nzero), pk(-1.0f), pk(K.hh3)));
        const f2 lB = mulr2(pk(-a.B, -lapB), lap, K.nzero);
        acc.cfl = fa(acc.cfl, lo(lB));
        acc.cfl = fa(acc.cfl, hi(lB));
        const f2 inv = pk(__frcp_rn(fmaxf(la, K.clamp)), __frcp_rn(fmaxf(lb, K.clamp)));
        const f2 d = fma2(L, pk(-1.0f), pk(K.h));  // h - |r|
        const f2 pw2 = mul2(d, d), cs = pk(K.cs);
        const f2 coef = mul2(pk(a.AA, b.AA), pk(K.mass));
        const f2 B = pk(a.B, b.B);
        const f2 lv = mul2(cs, d);
        const f2 pw = mul2(hs, hs);
        const f2 x = pk(a.x, b.x), y = pk(a.y, b.y), z = pk(a.z, b.z);
        const f2 gx = mulr2(coef, mul2(mul2(mul2(x, inv), cs), pw2), K.nzero);
        const f2 gy = mulr2(coef, mul2(mul2(mul2(y, inv), cs), pw2), K.nzero);
        const f2 gz = mulr2(coef, mul2(mul2(mul2(z, inv), cs), pw2), K.nzero);
        acc.fpx = fa(fa(acc.fpx, lo(gx)), hi(gx));
        acc.fpy = fa(fa(acc.fpy, lo(gy)), hi(gy));
        acc.fpz = fa(fa(acc.fpz, lo(gz)), hi(gz));
        const f2 vx = mulr2(mul2(pk(a.vx, b.vx), B), lv, K.nzero);
        const f2 vy = mulr2(mul2(pk(a.vy, b.vy), B), lv, K.nzero);
        const f2 vz = mulr2(mul2(pk(a.vz, b.vz), B), lv, K.nzero);
        acc.fvx = fa(fa(acc.fvx, lo(vx)), hi(vx));
        acc.fvy = fa(fa(acc.fvy, lo(vy)), hi(vy));
        acc.fvz = fa(fa(acc.fvz, lo(vz)), hi(vz));
        const f2 nx = mulr2(B, mul2(mul2(x, cg), pw), K.nzero);
        const f2 ny = mulr2(B, mul2(mul2(y, cg), pw), K.nzero);
        const f2 nz = mulr2(B, mul2(mul2(z, cg), pw), K.nzero);
        acc.nx = fa(fa(acc.nx, lo(nx)), hi(nx));
        acc.ny = fa(fa(acc.ny, lo(ny)), hi(ny));
        acc.nz = fa(fa(acc.nz, lo(nz)), hi(nz));
    }
}

template <bool FM>
__device__ __forceinline__ PairIn pair_in(const Rec& r, float nxi, float nyi, float nzi, float Ai, float nvx, float nvy,
                                          float nvz) {
    PairIn q;
    if (FM) {
        const f2 xy = add2(r.xy, pk(nxi, nyi)), zA = add2(r.zA, pk(nzi, Ai)), vxy = add2(r.vxy, pk(nvx, nvy));
        q.x = lo(xy), q.y = hi(xy), q.z = lo(zA), q.AA = hi(zA), q.vx = lo(vxy), q.vy = hi(vxy);
    } else {
        q.x = fa(lo(r.xy), nxi), q.y = fa(hi(r.xy), nyi), q.z = fa(lo(r.zA), nzi), q.AA = fa(hi(r.zA), Ai);
        q.vx = fa(lo(r.vxy), nvx), q.vy = fa(hi(r.vxy), nvy);
    }
    q.vz = fa(lo(r.vzB), nvz);
    q.B = hi(r.vzB);
    q.s = FM ? dist2_fma(q.x, q.y, q.z) : dist2(q.x, q.y, q.z);
    return q;
}

// One pair in the general form: the particle itself adds to the colour field
// only, a coincident neighbour takes the fixed direction.
template <bool FM>
__device__ __forceinline__ void force_one(const SceneDev& S, ForceAcc& acc, const PairIn& q, bool self) {
    const float4 dv = make_float4(q.vx, q.vy, q.vz, 0.0f);
    if (FM)
        force_pair_fast(S, acc, -q.x, -q.y, -q.z, q.s, 0.0f, 0.0f, 0.0f, q.AA, dv, 0.0f, q.B, -1, self);
    else
        force_pair(S, acc, -q.x, -q.y, -q.z, fsq(q.s), 0.0f, 0.0f, 0.0f, q.AA, dv, 0.0f, q.B, -1, self);
}

template <bool FM>
__device__ __noinline__ void force_cells(const DevArrays& a, const SceneDev& S, int p, ForceAcc& acc);

// force over the packed records: the list walk of k_force taken two
// neighbours at a time, in warp slices from the counter.  The L1 data path
// bounds it: a gather of 32 records from a few cells costs about 24 of its
// cycles, 71% of the fast form's time; taking neighbours in pairs cut the
// other part, the instructions (227 to 137 million a launch at 1,048,576
// particles, 56 in range), and with them the time from 351 to 270 us (exact
// arithmetic 447 to 364, with the packed records in place of three arrays);
// list entries read two to a load brought 240 and 353.  The fast form loads
// the records of the next pair before it sums the current one, at 80 registers
// and 24 warps an SM (without, entries still read one by one: 281 us at 64
// registers, 309 at 80); the exact form, with more arithmetic between its
// loads, is faster with 32 warps and no records in flight (364 vs 375 us).
template <bool FM, bool REC>
__global__ void __launch_bounds__(kMaxTile, FM ? 3 : 4) k_force_rec(const __grid_constant__ DevArrays a) {
    const int nwork = *a.n_ptiles;
    const int spt = a.tile / 32;
    for (int sl = first_slice<true>(a.ctr + 1); sl < nwork * spt; sl = next_slice<true>(a.ctr + 1, sl)) {
        const int w = sl / spt;
        const int li = (sl % spt) * 32 + (int)(threadIdx.x & 31);
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if ((S.flags & kFlagOrdered) != 0) continue;
        const int p = wk.start + li;
        if (p >= S.p_off + S.n) continue;
        const uint32_t pl = (uint32_t)(p - S.p_off);
        ForceAcc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
        const int cnt = a.ncnt[p];
        if (cnt <= kNbCap) {
            const float4* fd = a.fdat + 2 * (size_t)S.p_off;
            const uint32_t* nl = a.nlist + (size_t)wk.start * kNbCap + 4 * li;
            const uint32_t stride = 4 * a.tile;
            const PairConst K = {S.h, S.hh, FM ? 3.0f * S.hh : fm(fm(3.0f, S.h), S.h), S.c_grad, S.c_spiky, S.mass,
                                 FM ? S.cthr * S.cthr : S.cthr, neg_zero()};
            // pairs closer than the threshold (with a margin) take the general
            // form, and so do all pairs of a particle whose own velocity, or a
            // factor of its pair with itself, is not finite (zero times those
            // is not zero)
            const Rec me = ld_rec(fd + 2 * pl);
            const float nxi = -lo(me.xy), nyi = -hi(me.xy), nzi = -lo(me.zA), Ai = hi(me.zA);
            const float nvx = -lo(me.vxy), nvy = -hi(me.vxy), nvz = -lo(me.vzB);
            const float coef = (Ai + Ai) * K.mass;
            const float own = (FM ? coef * K.cs * (K.h * K.h) * rsqrtf(K.clamp) : coef) +
                              hi(me.vzB) * (K.h * K.cs) + hi(me.vzB) * K.cg * (K.hh * K.hh) + K.hh * K.cg * K.hh3;
            const bool odd = !((nvx + nvy + nvz) * 0.0f + own * 0.0f == 0.0f);
            const float c2 = odd ? INFINITY : S.cthr * S.cthr * 1.0001f;
            const bool rec = REC && (S.flags & kFlagRecord) != 0;
            // the list, two entries at a time; past its end: the particle itself
            uint32_t step = 2;  // to the next two: within the group of four, then to the next group
            auto two_at = [&](int q) {
                uint2 e = make_uint2(pl, pl);
                if (q < cnt) e = __ldg(reinterpret_cast<const uint2*>(nl));
                if (q + 1 >= cnt) e.y = pl;
                nl += step;
                step = stride - step;
                return e;
            };
            uint2 j = two_at(0), k = two_at(2);
            Rec ra, rb;
            if (FM) {
                ra = ld_rec(fd + 2 * j.x);
                rb = ld_rec(fd + 2 * j.y);
            }
            for (int q = 0; q < cnt; q += 2) {
                if (!FM) {
                    ra = ld_rec(fd + 2 * j.x);
                    rb = ld_rec(fd + 2 * j.y);
                }
                const PairIn A = pair_in<FM>(ra, nxi, nyi, nzi, Ai, nvx, nvy, nvz);
                const PairIn B = pair_in<FM>(rb, nxi, nyi, nzi, Ai, nvx, nvy, nvz);
                if (FM) {
                    ra = ld_rec(fd + 2 * k.x);
                    rb = ld_rec(fd + 2 * k.y);
                }
                bool general = false;
                if (fminf(A.s, B.s) < c2) general = odd || (A.s < c2 && j.x != pl) || (B.s < c2 && j.y != pl);
                if (REC && rec) {
                    const float4* sp = a.spos + S.p_off;
                    if (j.x != pl) acc.nb = max(acc.nb, __float_as_int(__ldg(&sp[j.x].w))), acc.any = 1;
                    if (j.y != pl) acc.nb = max(acc.nb, __float_as_int(__ldg(&sp[j.y].w))), acc.any = 1;
                }
                const bool two = q + 1 < cnt;
                if (!general) {
                    force_two<FM>(K, acc, A, B, two ? B.B : 0.0f);
                } else {
                    force_one<FM>(S, acc, A, j.x == pl);
                    if (two) force_one<FM>(S, acc, B, j.y == pl);
                }
                j = k;
                k = two_at(q + 4);
            }
        }
        const float4 xi = a.spos[p];
        const float4 vi = a.svel[p];
        const float4 di = a.dyn[p];
        if (cnt > kNbCap) {
            ForceAcc walk = acc;
            force_cells<FM>(a, S, p, walk);
            acc = walk;
        }
        integrate_and_store(a, S, p, xi, vi, di.x, acc, true);
    }
}

// ---------------------------------------------------------------------------
// Cooperative neighbour passes (variant bit 8): a group of G lanes shares one
// particle.  The lists the density pass hands to the force pass are
// particle-major here (particle p's entries at p * kNbCap + q), which both
// passes read and write in contiguous runs.

// Range [st, en) of stencil row r of the particle at probe q: rows in the
// order of for_rows (dz outer, dy inner, both ascending), trimmed the same
// way, so a particle's candidates come in the same order.  gx2 holds the
// squared x-gaps, in y/z cell units, of the x cells cx - 2 .. cx + 2 (R = 1
// with xsub 2, R = 2 with xsub 1; unused for R = 0, the general reach).
template <int R>
__device__ __forceinline__ void stencil_row(const DevArrays& a, const SceneDev& S, const Probe& q, const float* gx2,
                                            int r, uint32_t& st, uint32_t& en) {
    st = en = 0;
    const int side = R > 0 ? 2 * R + 1 : 2 * S.reach + 1;
    const int reach = R > 0 ? R : S.reach;
    const int dz = r / side - reach, dy = r % side - reach;
    const int z = q.c.cz + dz, y = q.c.cy + dy;
    if (!q.finite || z < 0 || z >= S.nz || y < 0 || y >= S.ny) return;
    const uint32_t* off = a.offsets + S.k_off;
    if (R > 0) {
        const float gz = cell_gap(q.tz, z, S.nz), gy = cell_gap(q.ty, y, S.ny);
        const float r2 = S.hcell * S.hcell - gy * gy - gz * gz;
        if (!(r2 >= 0.0f)) return;
        int lo = 0, hi = 0;
        constexpr int RX = (R > 0 ? R : 1) * (R == 1 ? 2 : 1);
#pragma unroll
        for (int d = 1; d <= RX; ++d) {
            if (gx2[RX - d] <= r2) lo = -d;
            if (gx2[RX + d] <= r2) hi = d;
        }
        const uint32_t row = row_key(a.tab, S, y, z);
        st = off[row + q.c.cx + lo];
        en = off[row + q.c.cx + hi + 1];
    } else {
        int xl, xh;
        if (!row_span(S, q, y, z, &xl, &xh)) return;
        const uint32_t row = row_key(a.tab, S, y, z);
        st = off[row + xl];
        en = off[row + xh + 1];
    }
}

// The neighbour sums of a particle whose list overflowed: it walks its cells
// (same order).  A call, so that this rare path takes no registers from the
// list walk.
template <bool FM>
__device__ __noinline__ void force_cells(const DevArrays& a, const SceneDev& S, int p, ForceAcc& acc) {
    const int pl = p - S.p_off;
    const float4 xi = a.spos[p], vi = a.svel[p], di = a.dyn[p];
    const float4* sp = a.spos + S.p_off;
    const float4* sv = a.svel + S.p_off;
    const float4* sd = a.dyn + S.p_off;
    const Probe q = probe_of(S, xi);
    const int side = 2 * S.reach + 1;
    for (int r = 0; r < side * side; ++r) {
        uint32_t st, en;
        stencil_row<0>(a, S, q, nullptr, r, st, en);
        for (uint32_t j = st; j < en; ++j) {
            const float4 xj = sp[j];
            const float rx = fs(xi.x, xj.x), ry = fs(xi.y, xj.y), rz = fs(xi.z, xj.z);
            const float s = dist2(rx, ry, rz);
            if (!(s <= S.smax)) continue;
            const float4 vj = sv[j], dj = sd[j];
            if (FM)
                force_pair_fast(S, acc, rx, ry, rz, dist2_fma(rx, ry, rz), vi.x, vi.y, vi.z, di.y, vj, dj.y, dj.z,
                                __float_as_int(xj.w), (int)j == pl);
            else
                force_pair(S, acc, rx, ry, rz, fsq(s), vi.x, vi.y, vi.z, di.y, vj, dj.y, dj.z, __float_as_int(xj.w),
                           (int)j == pl);
        }
    }
}

// Group geometry of G lanes per particle (G a power of two, 4..32).
template <int G>
struct Group {
    int gl;         // lane within the group
    int gbase;      // first lane of the group within the warp
    unsigned mask;  // the group's lanes
    __device__ __forceinline__ Group() {
        const int lane = threadIdx.x & 31;
        gl = lane & (G - 1);
        gbase = lane & ~(G - 1);
        mask = G == 32 ? kFull : (((1u << G) - 1u) << gbase);
    }
};

// Sum over the group, the same bits in every lane (each butterfly step adds
// two equal-rounded operands in either order), in a fixed order.
template <int G>
__device__ __forceinline__ float group_sum(float v, unsigned mask) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = fa(v, __shfl_xor_sync(mask, v, o, G));
    return v;
}

// density, cooperative: the group walks the particle's candidates as one
// stream (row after row, ascending index within a row) in windows of G, one
// candidate per lane, so neighbouring lanes load neighbouring particles.
// Each lane sums its candidates' terms in stream order; the group's partial
// sums are combined by group_sum.  In-range candidates are appended to the
// particle's list in stream order (ballot + prefix count).
template <int G, int R, bool PACK>
__device__ __forceinline__ void density_coop_particle(const DevArrays& a, const SceneDev& S, int p, int* soff,
                                                      const Group<G>& g) {
    const float4 xi = a.spos[p];
    const Probe q = probe_of(S, xi);
    constexpr int XS = R == 1 ? 2 : 1;  // the scene's xsub at this reach
    constexpr int RX = (R > 0 ? R : 1) * XS;
    float gx2[2 * RX + 1];  // squared x-gaps in y/z cell units
    if (R > 0) {
#pragma unroll
        for (int d = -RX; d <= RX; ++d) {
            const int k = q.c.cx + d;
            float g2 = INFINITY;
            if (k >= 0 && k < S.nx) {
                const float gg = cell_gap(q.tx, k, S.nx) * (1.0f / XS);
                g2 = gg * gg;
            }
            gx2[d + RX] = g2;
        }
    }
    const float4* sp = a.spos + S.p_off;
    uint32_t* nl = a.nlist + (size_t)p * kNbCap;
    const int side = R > 0 ? 2 * R + 1 : 2 * S.reach + 1;
    const int nrows = side * side;
    float rho = 0.0f;
    int cnt = 0;
    const unsigned below = (1u << g.gl) - 1u;
    for (int rb = 0; rb < nrows; rb += G) {
        uint32_t st = 0, en = 0;
        if (rb + g.gl < nrows) stencil_row<R>(a, S, q, gx2, rb + g.gl, st, en);
        const int len = (int)(en - st);
        int inc = len;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int v = __shfl_up_sync(g.mask, inc, o, G);
            if (g.gl >= o) inc += v;
        }
        const int pre = inc - len;
        const int total = __shfl_sync(g.mask, inc, G - 1, G);
        int carry = 0;
        for (int wb = 0; wb < total; wb += G) {
            // the rows that start in this window record where their
            // candidates sit: candidate t of the stream is particle t + off
            const bool starts = len > 0 && pre >= wb && pre < wb + G;
            if (starts) soff[pre - wb] = (int)st - pre;
            const unsigned m = __reduce_or_sync(g.mask, starts ? (1u << (pre - wb)) : 0u);
            __syncwarp(g.mask);
            const unsigned upto = m & ((2u << g.gl) - 1u);
            const int off = upto ? soff[31 - __clz(upto)] : carry;
            carry = m ? soff[31 - __clz(m)] : carry;
            __syncwarp(g.mask);
            const int t = wb + g.gl;
            bool in = false;
            uint32_t j = 0;
            float s = 0.0f;
            if (t < total) {
                j = (uint32_t)(t + off);
                const float4 xj = __ldg(sp + j);
                s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                in = s <= S.smax;
            }
            if (in) rho = fa(rho, density_term(S, fsq(s)));
            const unsigned b = (__ballot_sync(g.mask, in) & g.mask) >> g.gbase;
            const int at = cnt + __popc(b & below);
            if (in && at < kNbCap) nl[at] = j;
            cnt += __popc(b);
        }
    }
    rho = group_sum<G>(rho, g.mask);
    if (g.gl == 0) {
        const float P = fm(S.k, fs(rho, S.p0));
        const float Ai = fdv(P, fm(rho, rho)), Bi = fdv(S.mass, rho);
        a.dyn[p] = make_float4(rho, Ai, Bi, P);
        a.ncnt[p] = cnt;
        if (PACK) {
            const float4 vi = a.svel[p];
            a.fdat[2 * (size_t)p] = make_float4(xi.x, xi.y, xi.z, Ai);
            a.fdat[2 * (size_t)p + 1] = make_float4(vi.x, vi.y, vi.z, Bi);
        }
    }
}

template <int G, bool PACK>
__global__ void __launch_bounds__(256) k_density_coop(DevArrays a) {
    __shared__ int s_off[256];
    const Group<G> g;
    int* soff = s_off + (threadIdx.x & ~(G - 1));
    const int group = threadIdx.x / G, ngroups = blockDim.x / G;
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if (S.flags & kFlagOrdered) continue;
        const int end = min(wk.start + (int)blockDim.x, S.p_off + S.n);
        for (int p = wk.start + group; p < end; p += ngroups) {
            if (S.reach == 2)
                density_coop_particle<G, 2, PACK>(a, S, p, soff, g);
            else if (S.reach == 1)
                density_coop_particle<G, 1, PACK>(a, S, p, soff, g);
            else
                density_coop_particle<G, 0, PACK>(a, S, p, soff, g);
        }
    }
}

// force, cooperative: the group splits the particle's list (lane gl takes
// entries gl, gl + G, ...), each lane sums its pairs' terms in list order,
// the group combines them with group_sum, and every lane of the group then
// holds the particle's sums; the integration, contacts and erosion are
// computed alike in every lane and written by lane 0.  A particle whose list
// overflowed has the group split its cell rows instead (row r to lane r mod G).
template <int G, bool PACK, int MINB>
__global__ void __launch_bounds__(256, MINB) k_force_coop(DevArrays a) {
    const Group<G> g;
    const int group = threadIdx.x / G, ngroups = blockDim.x / G;
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if (S.flags & kFlagOrdered) continue;
        const int end = min(wk.start + (int)blockDim.x, S.p_off + S.n);
        for (int p = wk.start + group; p < end; p += ngroups) {
            const int pl = p - S.p_off;
            const float4 xi = a.spos[p];
            const float4 vi = a.svel[p];
            const float4 di = a.dyn[p];
            const float rho = di.x, Ai = di.y;
            ForceAcc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
            const float4* sp = a.spos + S.p_off;
            const float4* sv = a.svel + S.p_off;
            const float4* sd = a.dyn + S.p_off;
            const bool rec = (S.flags & kFlagRecord) != 0;
            auto pair = [&](uint32_t j, float4 xj, float4 vj, float Aj, float Bj, int idj) {
                const float rx = fs(xi.x, xj.x), ry = fs(xi.y, xj.y), rz = fs(xi.z, xj.z);
                force_pair(S, acc, rx, ry, rz, fsq(dist2(rx, ry, rz)), vi.x, vi.y, vi.z, Ai, vj, Aj, Bj, idj,
                           (int)j == pl);
            };
            const int cnt = a.ncnt[p];
            if (cnt <= kNbCap) {
                const uint32_t* nl = a.nlist + (size_t)p * kNbCap;
                int qn = g.gl;
                uint32_t j0 = qn < cnt ? __ldg(nl + qn) : 0u;
                for (int qq = g.gl; qq < cnt; qq += G) {
                    qn += G;
                    const uint32_t j1 = qn < cnt ? __ldg(nl + qn) : 0u;  // next entry, loaded ahead
                    if (PACK) {
                        const float4* fd = a.fdat + 2 * (size_t)S.p_off;
                        const float4 r0 = __ldg(fd + 2 * j0), r1 = __ldg(fd + 2 * j0 + 1);
                        const int idj = rec ? __float_as_int(__ldg(&sp[j0].w)) : 0;
                        pair(j0, r0, r1, r0.w, r1.w, idj);
                    } else {
                        const float4 xj = __ldg(sp + j0), vj = __ldg(sv + j0), dj = __ldg(sd + j0);
                        pair(j0, xj, vj, dj.y, dj.z, __float_as_int(xj.w));
                    }
                    j0 = j1;
                }
            } else {
                int r = 0;
                for_rows(a, S, xi, true, [&](uint32_t st, uint32_t en) {
                    if ((r++ & (G - 1)) != g.gl) return;
                    for (uint32_t j = st; j < en; ++j) {
                        const float4 xj = __ldg(sp + j);
                        if (dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z)) <= S.smax) {
                            const float4 vj = __ldg(sv + j), dj = __ldg(sd + j);
                            pair(j, xj, vj, dj.y, dj.z, __float_as_int(xj.w));
                        }
                    }
                });
            }
            acc.fpx = group_sum<G>(acc.fpx, g.mask);
            acc.fpy = group_sum<G>(acc.fpy, g.mask);
            acc.fpz = group_sum<G>(acc.fpz, g.mask);
            acc.fvx = group_sum<G>(acc.fvx, g.mask);
            acc.fvy = group_sum<G>(acc.fvy, g.mask);
            acc.fvz = group_sum<G>(acc.fvz, g.mask);
            acc.nx = group_sum<G>(acc.nx, g.mask);
            acc.ny = group_sum<G>(acc.ny, g.mask);
            acc.nz = group_sum<G>(acc.nz, g.mask);
            acc.cfl = group_sum<G>(acc.cfl, g.mask);
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                acc.nb = max(acc.nb, __shfl_xor_sync(g.mask, acc.nb, o, G));
                acc.any |= __shfl_xor_sync(g.mask, acc.any, o, G);
            }
            integrate_and_store(a, S, p, xi, vi, rho, acc, g.gl == 0);
        }
    }
}

// ---------------------------------------------------------------------------
// Neighbour passes for small systems: a group of G lanes per particle, as in
// the cooperative passes, but with every sum taken in list order, so that the
// results are the per-lane passes' bit for bit.  With one particle per lane a
// system of a few thousand particles is a few dozen warps, each walking its
// rows and lists as one chain of dependent loads; here the chain is one row
// table and a few windows of G candidates long.  The terms of a window are
// computed by all lanes and left in shared memory in order; the sequential
// additions, four cycles each, are then the only serial part, and one lane per
// particle does them and the per-particle arithmetic for the whole block.  All
// this takes about three times the per-lane passes' instructions, so it is for
// systems of few particles (group_rules).  Density and force, us, exact
// arithmetic: 1,000 particles 27 + 19 -> 10 + 10, 16,384 48 + 34 -> 25 + 20.
// Group number `slot` takes lane slot % T of work tile slot / T.
constexpr int kTerms = 256;  // density terms a group holds before it adds them

// The candidate stream of particle p, rows in traversal order, G candidates a
// window: window(in, j, s, id, b, cnt) receives in every lane of the group its
// candidate's index, squared distance and id, whether it is in range, the
// window's in-range lanes and the number in range before it.  Returns the
// number in range.
template <int G, int R, class F>
__device__ __forceinline__ int group_walk(const DevArrays& a, const SceneDev& S, float4 xi, int* soff, const Group<G>& g,
                                          F&& window) {
    const Probe q = probe_of(S, xi);
    constexpr int XS = R == 1 ? 2 : 1;  // the scene's xsub at this reach
    constexpr int RX = (R > 0 ? R : 1) * XS;
    float gx2[2 * RX + 1];  // squared x-gaps in y/z cell units
    if (R > 0) {
#pragma unroll
        for (int d = -RX; d <= RX; ++d) {
            const int k = q.c.cx + d;
            float g2 = INFINITY;
            if (k >= 0 && k < S.nx) {
                const float gg = cell_gap(q.tx, k, S.nx) * (1.0f / XS);
                g2 = gg * gg;
            }
            gx2[d + RX] = g2;
        }
    }
    const float4* sp = a.spos + S.p_off;
    const int side = R > 0 ? 2 * R + 1 : 2 * S.reach + 1;
    const int nrows = side * side;
    int cnt = 0;
    for (int rb = 0; rb < nrows; rb += G) {
        uint32_t st = 0, en = 0;
        if (rb + g.gl < nrows) stencil_row<R>(a, S, q, gx2, rb + g.gl, st, en);
        const int len = (int)(en - st);
        int inc = len;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int v = __shfl_up_sync(g.mask, inc, o, G);
            if (g.gl >= o) inc += v;
        }
        const int pre = inc - len;
        const int total = __shfl_sync(g.mask, inc, G - 1, G);
        int carry = 0;
        for (int wb = 0; wb < total; wb += G) {
            // the rows that start in this window record where their
            // candidates sit: candidate t of the stream is particle t + off
            const bool starts = len > 0 && pre >= wb && pre < wb + G;
            if (starts) soff[pre - wb] = (int)st - pre;
            const unsigned m = __reduce_or_sync(g.mask, starts ? (1u << (pre - wb)) : 0u);
            __syncwarp(g.mask);
            const unsigned upto = m & ((2u << g.gl) - 1u);
            const int off = upto ? soff[31 - __clz(upto)] : carry;
            carry = m ? soff[31 - __clz(m)] : carry;
            __syncwarp(g.mask);
            const int t = wb + g.gl;
            bool in = false;
            uint32_t j = 0;
            float s = 0.0f;
            int id = 0;
            if (t < total) {
                j = (uint32_t)(t + off);
                const float4 xj = sp[j];
                s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
                in = s <= S.smax;
                id = __float_as_int(xj.w);
            }
            const unsigned b = (__ballot_sync(g.mask, in) & g.mask) >> g.gbase;
            window(in, j, s, id, b, cnt);
            cnt += __popc(b);
        }
    }
    return cnt;
}

// The walk for the scene's reach.
template <int G, class F>
__device__ __forceinline__ int group_walk_any(const DevArrays& a, const SceneDev& S, float4 xi, int* soff,
                                              const Group<G>& g, F&& window) {
    if (S.reach == 1) return group_walk<G, 1>(a, S, xi, soff, g, window);
    if (S.reach == 2) return group_walk<G, 2>(a, S, xi, soff, g, window);
    return group_walk<G, 0>(a, S, xi, soff, g, window);
}

template <int G, int R, bool FM>
__device__ __forceinline__ void density_group_particle(const DevArrays& a, const SceneDev& S, int p, uint32_t* nl,
                                                       int stride, int* soff, float* term, const Group<G>& g,
                                                       int& count, int& left, float& part) {
    const float mc = S.mass * S.c_poly6;
    float rho = 0.0f;
    int done = 0;  // terms added
    auto make_terms = [&](int cnt) {  // squared distances to terms
        __syncwarp(g.mask);
        for (int k = g.gl; k < cnt - done; k += G) {
            const float hs = S.hh - term[k];
            term[k] = FM ? hs * hs * hs : density_term(S, fsq(term[k]));
        }
    };
    const unsigned below = (1u << g.gl) - 1u;
    const int cnt = group_walk<G, R>(a, S, a.spos[p], soff, g, [&](bool in, uint32_t j, float s, int, unsigned b, int n) {
        if (n - done > kTerms - G) {
            make_terms(n);
            __syncwarp(g.mask);
            for (int k = 0; k < n - done; ++k) rho = FM ? fmaf(mc, term[k], rho) : fa(rho, term[k]);
            done = n;
            __syncwarp(g.mask);
        }
        if (in) {
            const int at = n + __popc(b & below);
            if (nl && at < kNbCap) nl[(size_t)(at >> 2) * stride + (at & 3)] = j;
            term[at - done] = s;
        }
    });
    make_terms(cnt);
    count = cnt;
    left = cnt - done;
    part = rho;
}

// lane_lists: the lists (and the packed records) go to a per-lane force pass;
// else a list's entries are together, for k_force_group.  Each warp takes one
// particle; one lane for each of the block's particles then adds its terms and
// finishes it.
template <bool FM>
__global__ void __launch_bounds__(256, 5) k_density_group(const __grid_constant__ DevArrays a, bool lane_lists,
                                                          bool pack) {
    step_enter(a.early);
    constexpr int G = 32, N = 256 / G;
    __shared__ int s_off[256];
    __shared__ float s_term[N][kTerms + 1];
    __shared__ int s_p[N], s_cnt[N], s_left[N];
    __shared__ float s_part[N];
    const Group<G> g;
    const int wid = threadIdx.x / G, slot = (int)blockIdx.x * N + wid, w = slot / a.tile, l = slot % a.tile;
    Work wk = {0, 0};
    int p = -1;
    if (w < *a.n_ptiles) {
        wk = a.ptiles[w];
        const SceneDev& S = a.scenes[wk.scene];
        if (a.steps_left[wk.scene] != 0 && !(S.flags & kFlagOrdered) && wk.start + l < S.p_off + S.n) p = wk.start + l;
    }
    const SceneDev& S = a.scenes[wk.scene];  // the tile's, the same for the whole block
    if (p >= 0) {
        int* soff = s_off + (threadIdx.x & ~(G - 1));
        float* term = s_term[wid];
        const int stride = 4 * (lane_lists ? a.tile : 1);
        uint32_t* nl = a.nlist ? a.nlist + (lane_lists ? (size_t)wk.start * kNbCap + 4 * l : (size_t)p * kNbCap) : nullptr;
        int cnt, left;
        float part;
        if (S.reach == 1)
            density_group_particle<G, 1, FM>(a, S, p, nl, stride, soff, term, g, cnt, left, part);
        else if (S.reach == 2)
            density_group_particle<G, 2, FM>(a, S, p, nl, stride, soff, term, g, cnt, left, part);
        else
            density_group_particle<G, 0, FM>(a, S, p, nl, stride, soff, term, g, cnt, left, part);
        if (g.gl == 0) s_cnt[wid] = cnt, s_left[wid] = left, s_part[wid] = part;
    }
    if (g.gl == 0) s_p[wid] = p;
    __syncthreads();
    const int q = threadIdx.x;
    if (q >= N || s_p[q] < 0) return;
    p = s_p[q];
    const float mc = S.mass * S.c_poly6;
    float rho = s_part[q];
    for (int k = 0; k < s_left[q]; ++k) rho = FM ? fmaf(mc, s_term[q][k], rho) : fa(rho, s_term[q][k]);
    const float P = fm(S.k, fs(rho, S.p0));
    const float Ai = fdv(P, fm(rho, rho)), Bi = fdv(S.mass, rho);
    a.dyn[p] = make_float4(rho, Ai, Bi, P);
    if (a.ncnt) a.ncnt[p] = s_cnt[q];
    if (pack) {
        const float4 xi = a.spos[p], vi = a.svel[p];
        a.fdat[2 * (size_t)p] = make_float4(xi.x, xi.y, xi.z, Ai);
        a.fdat[2 * (size_t)p + 1] = make_float4(vi.x, vi.y, vi.z, Bi);
    }
}

// Values a lane leaves for the ordered sums of one pair.  Exact arithmetic:
// the ten addends (pressure, viscosity, normal, colour field).  Fast: the
// factors of the ten fused multiply-adds: the pressure direction, r, the
// velocity difference, then g, b, gn, m/rho_j and the Laplacian.
template <bool FM>
constexpr int kPairValues = FM ? 14 : 10;

template <bool FM>
__device__ __forceinline__ void pair_values(const SceneDev& S, float rx, float ry, float rz, float vx, float vy, float vz,
                                            float AA, float Bj, bool self, float* v) {
#pragma unroll
    for (int c = 0; c < kPairValues<FM>; ++c) v[c] = 0.0f;  // the particle itself adds to the colour field only
    if (FM) {
        const float s = dist2_fma(rx, ry, rz);
        const float hs = S.hh - s;
        v[12] = Bj;
        v[13] = (-S.c_grad * hs) * fmaf(-7.0f, s, 3.0f * S.hh);
        if (self) return;
        const float coef = AA * S.mass;
        if (s < S.cthr * S.cthr) {
            const float hl = S.h - sqrtf(s);
            const float t = -(S.inv_sqrt3 * S.c_spiky) * (hl * hl);
            v[0] = v[1] = v[2] = coef;
            v[9] = t;
            v[10] = Bj * (S.c_spiky * hl);
        } else {
            const float inv = rsqrtf(s);
            const float hl = fmaf(-s, inv, S.h);
            v[0] = rx, v[1] = ry, v[2] = rz;
            v[9] = -(S.c_spiky * coef) * (hl * hl) * inv;
            v[10] = Bj * (S.c_spiky * hl);
        }
        v[3] = rx, v[4] = ry, v[5] = rz;
        v[6] = vx, v[7] = vy, v[8] = vz;
        v[11] = -(Bj * S.c_grad) * (hs * hs);
    } else {
        // one pair from zero sums: 0 + x is x (a zero's sign aside)
        ForceAcc one = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
        force_pair(S, one, rx, ry, rz, fsq(dist2(rx, ry, rz)), 0.f, 0.f, 0.f, AA, make_float4(vx, vy, vz, 0.f), 0.f, Bj,
                   -1, self);
        v[0] = one.fpx, v[1] = one.fpy, v[2] = one.fpz;
        v[3] = one.fvx, v[4] = one.fvy, v[5] = one.fvz;
        v[6] = one.nx, v[7] = one.ny, v[8] = one.nz;
        v[9] = one.cfl;
    }
}

template <bool FM, bool REC>
__global__ void __launch_bounds__(256, 4) k_force_group(const __grid_constant__ DevArrays a) {
    step_enter(a.early);
    constexpr int G = 16, N = 256 / G, V = kPairValues<FM>, W = G + 1;
    __shared__ float s_val[N][V][W];
    __shared__ float s_sum[N][13];  // the ten sums, NeighbId, whether there is a neighbour; the particle
    const Group<G> g;
    const int grp = threadIdx.x / G, slot = (int)blockIdx.x * N + grp, w = slot / a.tile;
    float(*val)[W] = s_val[grp];
    float* sum = s_sum[grp];
    Work wk = {0, 0};
    int p = -1;
    if (w < *a.n_ptiles) {
        wk = a.ptiles[w];
        const SceneDev& S = a.scenes[wk.scene];
        const int at = wk.start + slot % a.tile;
        if (a.steps_left[wk.scene] != 0 && !(S.flags & kFlagOrdered) && at < S.p_off + S.n) p = at;
    }
    const SceneDev& S = a.scenes[wk.scene];  // the tile's, the same for the whole block
    const int cnt = p >= 0 ? a.ncnt[p] : 0;
    int nb = -1, any = 0;
    if (p < 0) {
    } else if (cnt > kNbCap) {  // the list overflowed: one lane walks the cells
        if (g.gl == 0) {
            ForceAcc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
            force_cells<FM>(a, S, p, acc);
            sum[0] = acc.fpx, sum[1] = acc.fpy, sum[2] = acc.fpz;
            sum[3] = acc.fvx, sum[4] = acc.fvy, sum[5] = acc.fvz;
            sum[6] = acc.nx, sum[7] = acc.ny, sum[8] = acc.nz;
            sum[9] = acc.cfl;
            nb = acc.nb, any = acc.any;
        }
    } else {
        const float4 xi = a.spos[p], vi = a.svel[p];
        const float Ai = a.dyn[p].y;
        const uint32_t pl = (uint32_t)(p - S.p_off);
        const float4* sp = a.spos + S.p_off;
        const float4* sv = a.svel + S.p_off;
        const float4* sd = a.dyn + S.p_off;
        const uint32_t* nl = a.nlist + (size_t)p * kNbCap;
        // the two factors (or the addend) of this lane's sum
        const int c = g.gl;
        const int i1 = FM ? (c < 3 ? c : c < 6 ? c + 3 : c < 9 ? c - 3 : 12) : c;
        const int i2 = c < 3 ? 9 : c < 6 ? 10 : c < 9 ? 11 : 13;
        float acc = 0.0f;
        uint32_t j = c < cnt ? nl[c] : pl;
        for (int b = 0; b < cnt; b += G) {
            const float4 xj = sp[j], vj = sv[j], dj = sd[j];
            const bool live = b + c < cnt, self = j == pl;
            if (REC && live && !self) nb = max(nb, __float_as_int(xj.w)), any = 1;
            if (b + G + c < cnt) j = nl[b + G + c];
            if (live) {
                float v[V];
                pair_values<FM>(S, fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z), fs(vj.x, vi.x), fs(vj.y, vi.y),
                                fs(vj.z, vi.z), fa(Ai, dj.y), dj.z, self, v);
#pragma unroll
                for (int k = 0; k < V; ++k) val[k][c] = v[k];
            }
            __syncwarp(g.mask);
            if (c < 10) {
                const int m = min(G, cnt - b);
                for (int k = 0; k < m; ++k) acc = FM ? fmaf(val[i1][k], val[i2][k], acc) : fa(acc, val[i1][k]);
            }
            __syncwarp(g.mask);
        }
        if (REC) {
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                nb = max(nb, __shfl_xor_sync(g.mask, nb, o, G));
                any |= __shfl_xor_sync(g.mask, any, o, G);
            }
        }
        if (c < 10) sum[c] = acc;
    }
    if (g.gl == 0) {
        sum[10] = __int_as_float(nb), sum[11] = __int_as_float(any);
        sum[12] = __int_as_float(p);
    }
    // one lane for each of the block's particles: the rest of the step
    __syncthreads();
    if (threadIdx.x >= N) return;
    sum = s_sum[threadIdx.x];
    p = __float_as_int(sum[12]);
    if (p < 0) return;
    const ForceAcc acc = {sum[0], sum[1], sum[2], sum[3], sum[4], sum[5], sum[6], sum[7], sum[8], sum[9],
                          __float_as_int(sum[10]), __float_as_int(sum[11])};
    integrate_and_store(a, S, p, a.spos[p], a.svel[p], a.dyn[p].x, acc, true);
}

// Ordered (validation) passes, a warp per particle: the in-range candidates of
// the walk are ranked by id, every lane counting the smaller ids of up to four
// of them, and the terms then added in rank order, which is the reference's
// order of summation (j ascending).  One lane per particle, sorting its list
// by insertion in local memory, takes 59 + 67 us for 5,000 particles; these 16 +
// 18 (group_rules).
struct OrderedList {
    uint32_t j[kMaxNb];
    int id[kMaxNb];
    float s[kMaxNb];
};

// Collects and ranks: lane gl's candidates gl, gl + 32, ... have the ranks
// rank[0], rank[1], ...  Returns the number in the list; more in range than it
// holds sets the status bit.
__device__ __forceinline__ int ordered_collect(const DevArrays& a, const SceneDev& S, float4 xi, int* soff,
                                               OrderedList& l, const Group<32>& g, int* rank) {
    const unsigned below = (1u << g.gl) - 1u;
    const int cnt = group_walk_any<32>(a, S, xi, soff, g, [&](bool in, uint32_t j, float s, int id, unsigned b, int n) {
        const int at = n + __popc(b & below);
        if (in && at < kMaxNb) l.j[at] = j, l.id[at] = id, l.s[at] = s;
    });
    const int m = min(cnt, kMaxNb);
    if (cnt > kMaxNb && g.gl == 0) atomicOr(a.status, 1u);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kMaxNb / 32; ++u) {
        const int k = g.gl + 32 * u;
        rank[u] = 0;
        if (k < m) {
            const int id = l.id[k];
            for (int q = 0; q < m; ++q) rank[u] += l.id[q] < id || (l.id[q] == id && l.j[q] < l.j[k]) ? 1 : 0;
        }
    }
    return m;
}

// The particle of warp `wid` of a block of 8 in tile order; -1: none.
__device__ __forceinline__ int ordered_particle(const DevArrays& a, int wid, Work& wk) {
    const int slot = (int)blockIdx.x * 8 + wid, w = slot / a.tile;
    wk = Work{0, 0};
    if (w >= *a.n_ptiles) return -1;
    wk = a.ptiles[w];
    const SceneDev& S = a.scenes[wk.scene];
    const int p = wk.start + slot % a.tile;
    return a.steps_left[wk.scene] != 0 && (S.flags & kFlagOrdered) && p < S.p_off + S.n ? p : -1;
}

__global__ void __launch_bounds__(256) k_density_ordered(const __grid_constant__ DevArrays a) {
    step_enter(a.early);
    __shared__ int s_off[8][32];
    __shared__ OrderedList s_list[8];
    const Group<32> g;
    const int wid = threadIdx.x >> 5;
    Work wk;
    const int p = ordered_particle(a, wid, wk);
    if (p < 0) return;
    const SceneDev& S = a.scenes[wk.scene];
    OrderedList& l = s_list[wid];
    int rank[kMaxNb / 32];
    const int m = ordered_collect(a, S, a.spos[p], s_off[wid], l, g, rank);
    float t[kMaxNb / 32];
#pragma unroll
    for (int u = 0; u < kMaxNb / 32; ++u)
        if (g.gl + 32 * u < m) t[u] = density_term(S, fsq(l.s[g.gl + 32 * u]));
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kMaxNb / 32; ++u)
        if (g.gl + 32 * u < m) l.s[rank[u]] = t[u];
    __syncwarp();
    float rho = 0.0f;
    for (int k = 0; k < m; ++k) rho = fa(rho, l.s[k]);
    if (g.gl == 0) {
        const float P = fm(S.k, fs(rho, S.p0));
        a.dyn[p] = make_float4(rho, fdv(P, fm(rho, rho)), fdv(S.mass, rho), P);
    }
}

__global__ void __launch_bounds__(256) k_force_ordered(const __grid_constant__ DevArrays a) {
    step_enter(a.early);
    constexpr int V = kPairValues<false>;
    __shared__ int s_off[8][32];
    __shared__ OrderedList s_list[8];
    __shared__ float s_val[8][V][33];
    __shared__ float s_sum[8][13];  // the ten sums, NeighbId, whether there is a neighbour; the particle
    const Group<32> g;
    const int wid = threadIdx.x >> 5;
    Work wk;
    int p = ordered_particle(a, wid, wk);
    const SceneDev& S = a.scenes[wk.scene];  // the tile's, the same for the whole block
    if (p >= 0) {
        OrderedList& l = s_list[wid];
        const float4 xi = a.spos[p], vi = a.svel[p];
        const float Ai = a.dyn[p].y;
        int rank[kMaxNb / 32];
        const int m = ordered_collect(a, S, xi, s_off[wid], l, g, rank);
        uint32_t jr[kMaxNb / 32];
#pragma unroll
        for (int u = 0; u < kMaxNb / 32; ++u)
            if (g.gl + 32 * u < m) jr[u] = l.j[g.gl + 32 * u];
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kMaxNb / 32; ++u)
            if (g.gl + 32 * u < m) l.j[rank[u]] = jr[u];
        __syncwarp();
        const uint32_t pl = (uint32_t)(p - S.p_off);
        float acc = 0.0f;
        int nb = -1, any = 0;
        for (int b = 0; b < m; b += 32) {
            if (b + g.gl < m) {
                const uint32_t j = l.j[b + g.gl];
                const float4 xj = a.spos[S.p_off + j], vj = a.svel[S.p_off + j], dj = a.dyn[S.p_off + j];
                if (j != pl) nb = max(nb, __float_as_int(xj.w)), any = 1;
                float v[V];
                pair_values<false>(S, fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z), fs(vj.x, vi.x), fs(vj.y, vi.y),
                                   fs(vj.z, vi.z), fa(Ai, dj.y), dj.z, j == pl, v);
#pragma unroll
                for (int k = 0; k < V; ++k) s_val[wid][k][g.gl] = v[k];
            }
            __syncwarp();
            if (g.gl < 10)
                for (int k = 0; k < min(32, m - b); ++k) acc = fa(acc, s_val[wid][g.gl][k]);
            __syncwarp();
        }
        nb = __reduce_max_sync(kFull, nb);
        any = __reduce_max_sync(kFull, any);
        if (g.gl < 10) s_sum[wid][g.gl] = acc;
        if (g.gl == 0) s_sum[wid][10] = __int_as_float(nb), s_sum[wid][11] = __int_as_float(any);
    }
    if (g.gl == 0) s_sum[wid][12] = __int_as_float(p);
    __syncthreads();
    if (threadIdx.x >= 8) return;
    const float* sum = s_sum[threadIdx.x];
    p = __float_as_int(sum[12]);
    if (p < 0) return;
    const ForceAcc acc = {sum[0], sum[1], sum[2], sum[3], sum[4], sum[5], sum[6], sum[7], sum[8], sum[9],
                          __float_as_int(sum[10]), __float_as_int(sum[11])};
    integrate_and_store(a, S, p, a.spos[p], a.svel[p], a.dyn[p].x, acc, true);
}

// ---------------------------------------------------------------------------
// Force pass with a TMA gather pipeline (variant bit 18, with lists, packed
// records and fast arithmetic).  Each block holds T consumer threads (one
// particle of the tile each) and one producer warp.  For list slot q the
// producer reads the T list entries (16-byte loads), keeps them in an index
// ring in shared memory and issues TMA tile::gather4 copies of the T packed
// records (rows of a 2-D tensor map over fdat, one row high) into a ring of
// stages in shared memory; each stage's copies complete on its `full`
// mbarrier, and the consumer warps release the stage through its `empty`
// mbarrier.  The consumers then sum the same pairs in the same order as the
// per-lane fast-arithmetic pass (the same bits), but their neighbour records
// come from shared memory and hold no registers while in flight.  Every wait
// is bounded by a clock limit; a wait that runs out sets status bit 2 and
// ends the block's work.
constexpr int kTmaRingBytes = 32768;  // record ring; stages = kTmaRingBytes / (T * 32)
constexpr long long kWaitLimit = 4000000000LL;  // clock cycles (about 2 s)

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Waits until the phase of parity `parity` has completed; false when the
// clock limit runs out first.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    const long long t0 = clock64();
    for (;;) {
        unsigned done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > kWaitLimit) return false;
    }
}

// Four rows (record indices) of the tensor map into 128 contiguous bytes of
// shared memory; rows outside the tensor read as zeros.
__device__ __forceinline__ void tma_gather4(void* dst, const CUtensorMap* map, int r0, int r1, int r2, int r3,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
        "%3, %4, %5, %6}], [%7];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(smem_u32(bar))
        : "memory");
}

template <int MINB>
__global__ void __launch_bounds__(kMaxTile + 32, MINB) k_force_tma(DevArrays a, const __grid_constant__ CUtensorMap fmap) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ int s_m;
    const int T = (int)blockDim.x - 32;  // consumers: 128 or 256
    const int D = kTmaRingBytes / (T * 32);
    unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);  // TMA wants 128-B rows
    float4* ring = reinterpret_cast<float4*>(smem);  // stage s, lane l: ring[2 * (s * T + l) + {0, 1}]
    uint32_t* jring = reinterpret_cast<uint32_t*>(smem + kTmaRingBytes);  // stage s, lane l: jring[s * T + l]
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kTmaRingBytes + (size_t)D * T * 4);
    uint64_t* empty = full + D;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool producer = tid >= T;
    if (tid == 0) {
        for (int q = 0; q < D; ++q) {
            mbar_init(full + q, 1);
            mbar_init(empty + q, (unsigned)(T / 32));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    unsigned it = 0;  // ring slots this block has used
    bool ok = true;
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        if (S.flags & kFlagOrdered) continue;
        const int end = S.p_off + S.n;
        if (producer) {
            int m = 0;
            for (int l = lane; l < T; l += 32) {
                const int p = wk.start + l;
                if (p < end) m = max(m, min(a.ncnt[p], kNbCap));
            }
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFull, m, o));
            if (lane == 0) s_m = ok ? m : 0;
        }
        __syncthreads();
        const int M = s_m;  // list slots in use in this tile
        if (producer) {
            const uint32_t* nl = a.nlist + (size_t)wk.start * kNbCap;
            const int per = T / 32;  // consumer lanes per producer lane
            for (int q = 0; q < M && ok; ++q) {
                const unsigned i2 = it + (unsigned)q, st = i2 % (unsigned)D, ph = (i2 / (unsigned)D) & 1u;
                if (i2 >= (unsigned)D && !mbar_wait(empty + st, ph ^ 1u)) {
                    ok = false;
                    break;
                }
                uint4 jj[2];
                for (int g = 0; g < per; g += 4) {
                    const uint32_t* e = nl + list_at(q, per * lane + g, T);
                    jj[g / 4] = make_uint4(e[0], e[4], e[8], e[12]);
                    *reinterpret_cast<uint4*>(jring + (size_t)st * T + per * lane + g) = jj[g / 4];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_expect_tx(full + st, (unsigned)(T * 32));
                for (int g = 0; g < per; g += 4) {
                    const uint4 v = jj[g / 4];
                    tma_gather4(ring + 2 * ((size_t)st * T + per * lane + g), &fmap, S.p_off + (int)v.x,
                                S.p_off + (int)v.y, S.p_off + (int)v.z, S.p_off + (int)v.w, full + st);
                }
            }
        } else {
            const int p0 = wk.start + tid;
            const bool valid = p0 < end;
            const int p = valid ? p0 : S.p_off;
            const int pl = p - S.p_off;
            const float4 xi = a.spos[p];
            const float4 vi = a.svel[p];
            const float4 di = a.dyn[p];
            const float rho = di.x, Ai = di.y;
            const int cnt = valid ? a.ncnt[p] : 0;
            const bool listed = cnt <= kNbCap;
            const bool rec = (S.flags & kFlagRecord) != 0;
            const float4* sp = a.spos + S.p_off;
            ForceAcc acc = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1, 0};
            for (int q = 0; q < M; ++q) {
                const unsigned i2 = it + (unsigned)q, st = i2 % (unsigned)D, ph = (i2 / (unsigned)D) & 1u;
                if (ok && !mbar_wait(full + st, ph)) ok = false;
                if (ok && listed && q < cnt) {
                    const float4 r0 = ring[2 * ((size_t)st * T + tid)], r1 = ring[2 * ((size_t)st * T + tid) + 1];
                    const uint32_t j = jring[(size_t)st * T + tid];
                    const int idj = rec ? __float_as_int(__ldg(&sp[j].w)) : 0;
                    const float rx = fs(xi.x, r0.x), ry = fs(xi.y, r0.y), rz = fs(xi.z, r0.z);
                    force_pair_fast(S, acc, rx, ry, rz, dist2_fma(rx, ry, rz), vi.x, vi.y, vi.z, Ai, r1, r0.w, r1.w, idj,
                                    (int)j == pl);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + st);
            }
            if (valid && !listed) {
                // the list overflowed: this lane walks its cells (same order)
                const float4* sv = a.svel + S.p_off;
                const float4* sd = a.dyn + S.p_off;
                for_each_candidate(a, S, xi, [&](uint32_t j, float4 xj) {
                    const float rx = fs(xi.x, xj.x), ry = fs(xi.y, xj.y), rz = fs(xi.z, xj.z);
                    if (dist2(rx, ry, rz) <= S.smax) {
                        const float4 vj = __ldg(sv + j), dj = __ldg(sd + j);
                        force_pair_fast(S, acc, rx, ry, rz, dist2_fma(rx, ry, rz), vi.x, vi.y, vi.z, Ai, vj, dj.y, dj.z,
                                        __float_as_int(xj.w), (int)j == pl);
                    }
                });
            }
            if (valid) integrate_and_store(a, S, p, xi, vi, rho, acc, true);
        }
        it += (unsigned)M;
        __syncthreads();
    }
    if (!ok) atomicOr(a.status, 4u);
}

size_t force_tma_smem(int tile) {
    const int D = kTmaRingBytes / (tile * 32);
    return 128 + kTmaRingBytes + (size_t)D * tile * 4 + 2 * (size_t)D * 8;
}

// terrain: height snapshot = base + delta * unit, read by the next step.
// Four vertices per thread: a tile of T vertices takes T / 4 threads, each
// with 16-byte loads and stores (a scene's vertices start on a 512-vertex
// boundary, so every thread's first vertex is 4-aligned).  A block takes 1024 /
// T tiles: with one tile, a warp or two, the blocks' own overhead was a third
// of the time (16.8 million vertices, tile 128: 72 -> 45 us, 5.96 TB/s of 16 B a
// vertex).
__global__ void __launch_bounds__(256) k_terrain(DevArrays a) {
    step_enter(a.early);
    const int nwork = *a.n_ttiles, T4 = a.tile / 4, per = 256 / T4;
    const int sub = threadIdx.x / T4, lane = threadIdx.x % T4;
    for (int w = blockIdx.x * per + sub; w < nwork; w += gridDim.x * per) {
        const Work wk = a.ttiles[w];
        if (a.steps_left[wk.scene] == 0) continue;
        const SceneDev& S = a.scenes[wk.scene];
        const int t = wk.start + 4 * lane;
        const int end = S.t_off + S.tw * S.td;
        const float u = S.height_unit;
        if (t + 3 < end) {
            const float4 b = *reinterpret_cast<const float4*>(a.tbase + t);
            const longlong2 d0 = *reinterpret_cast<const longlong2*>(a.tdelta + t);
            const longlong2 d1 = *reinterpret_cast<const longlong2*>(a.tdelta + t + 2);
            *reinterpret_cast<float4*>(a.theight + t) =
                make_float4(fa(b.x, fm(__ll2float_rn(d0.x), u)), fa(b.y, fm(__ll2float_rn(d0.y), u)),
                            fa(b.z, fm(__ll2float_rn(d1.x), u)), fa(b.w, fm(__ll2float_rn(d1.y), u)));
        } else {
            for (int k = t; k < end && k < t + 4; ++k) a.theight[k] = fa(a.tbase[k], fm(__ll2float_rn(a.tdelta[k]), u));
        }
    }
}

__global__ void k_tick(int* steps_left, int nscenes, bool early) {
    step_enter(early);
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nscenes && steps_left[s] > 0) steps_left[s] -= 1;
}

__global__ void __launch_bounds__(kMaxTile) k_neighbour_counts(DevArrays a, int32_t* out) {
    const int nwork = *a.n_ptiles;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const Work wk = a.ptiles[w];
        const SceneDev& S = a.scenes[wk.scene];
        const int p = wk.start + threadIdx.x;
        if (p >= S.p_off + S.n) continue;
        const float4 xi = a.spos[p];
        const int pl = p - S.p_off;
        int cnt = 0;
        for_each_candidate(a, S, xi, [&](uint32_t j, float4 xj) {
            float s = dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z));
            if (s <= S.smax && (int)j != pl) ++cnt;
        });
        const int id = __float_as_int(xi.w);
        if (id >= 0 && id < S.n) out[S.p_off + id] = cnt;
    }
}

// splitmix64's finaliser (Steele, Lea and Flood, "Fast splittable
// pseudorandom number generators", OOPSLA 2014).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ unsigned long long pair64(float lo, float hi) {
    return (unsigned long long)(uint32_t)__float_as_int(lo) |
           ((unsigned long long)(uint32_t)__float_as_int(hi) << 32);
}

// FP64 diagnostics: kDiagBlocks blocks per listed scene write fixed-order
// partial sums of momentum and energies (so the result is reproducible);
// integer totals use int64 atomics, which are exact in any order: sediment
// and terrain units, non-finite positions and the state fingerprint (sum of
// a mix of each particle's id and state bits, so any order of the particles
// in memory gives the same value).  isums holds three values per listed
// scene.
__global__ void __launch_bounds__(256) k_diag(DevArrays a, double* partial, long long* isums, int* nan_count) {
    __shared__ double sh[kDiagDoubles][8];
    const int li = blockIdx.x / kDiagBlocks, b = blockIdx.x % kDiagBlocks;
    const int sidx = a.scene_list[li];
    const SceneDev& S = a.scenes[sidx];
    double acc[kDiagDoubles] = {0, 0, 0, 0, 0, 0, 0, 0};
    long long sed = 0, ter = 0;
    unsigned long long fp = 0;
    int nan = 0;
    const double m = (double)S.mass;
    for (int q = b * 256 + threadIdx.x; q < S.n; q += kDiagBlocks * 256) {
        const float4 x = a.pos[S.p_off + q];
        const float4 v = a.vel[S.p_off + q];
        unsigned long long h = mix64(0x9e3779b97f4a7c15ULL * (unsigned long long)(uint32_t)(__float_as_int(x.w) + 1));
        h = mix64(h ^ pair64(x.x, x.y));
        h = mix64(h ^ pair64(x.z, v.x));
        h = mix64(h ^ pair64(v.y, v.z));
        h = mix64(h ^ (unsigned long long)(uint32_t)__float_as_int(v.w));
        fp += h;
        const double vx = v.x, vy = v.y, vz = v.z;
        acc[0] += m * vx;
        acc[1] += m * vy;
        acc[2] += m * vz;
        acc[3] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        acc[4] += -m * ((double)S.g[0] * x.x + (double)S.g[1] * x.y + (double)S.g[2] * x.z);
        sed += (long long)__float_as_int(v.w);
        if (!isfinite(x.x) || !isfinite(x.y) || !isfinite(x.z)) ++nan;
    }
    if (S.flags & kFlagTerrain)
        for (int t = b * 256 + threadIdx.x; t < S.tw * S.td; t += kDiagBlocks * 256) ter += a.tdelta[S.t_off + t];
    for (int c = 0; c < kDiagDoubles; ++c) {
        double v = acc[c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
        if ((threadIdx.x & 31) == 0) sh[c][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < kDiagDoubles) {
        double v = 0.0;
        for (int q = 0; q < 8; ++q) v += sh[threadIdx.x][q];
        partial[(size_t)blockIdx.x * kDiagDoubles + threadIdx.x] = v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        sed += __shfl_down_sync(kFull, sed, o);
        ter += __shfl_down_sync(kFull, ter, o);
        fp += __shfl_down_sync(kFull, fp, o);
        nan += __shfl_down_sync(kFull, nan, o);
    }
    if ((threadIdx.x & 31) == 0) {
        unsigned long long* u = reinterpret_cast<unsigned long long*>(isums + 3 * li);
        if (sed) atomicAdd(u, (unsigned long long)sed);
        if (ter) atomicAdd(u + 1, (unsigned long long)ter);
        if (fp) atomicAdd(u + 2, fp);
        if (nan) atomicAdd(nan_count + li, nan);
    }
}

// Launch of a kernel of the step (step_enter); early: with programmatic
// serialization.  It hides a kernel's launch behind the one before it: of
// 18,432 particles or less a step takes about 9 us less launched by itself (4
// steps of 1,000 124 vs 87 us) and 1 to 2 in a graph (64 steps 1,385 vs 1,275).  In large systems blocks that wait cost more than that (a step,
// us, with and without: 100,000 particles 127 vs 113, 1,048,576 862 vs 818,
// 8.4M 5,367 vs 4,949): the list passes keep the L1 split of the kernel they
// overlapped.
template <class T>
T with_early(T v, bool) {
    return v;
}
DevArrays with_early(DevArrays a, bool early) {
    a.early = early;  // tells the kernel to wait
    return a;
}
template <class... P, class... A>
void launch(bool early, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
    if (!early) {
        k<<<grid, block, smem, st>>>(P(with_early(args, early))...);
        return;
    }
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, k, P(with_early(args, early))...);
}

}  // namespace

void launch_sort_small(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_sort_small, s.grid_sort, kSortThreads, s.sort_smem, st, a);
}
size_t sort_small_smem(int64_t max_n, int64_t max_keys) {
    const int64_t per = ((max_keys + kSortThreads - 1) / kSortThreads) | 1;
    const int64_t bytes = (kSmallSort + per * kSortThreads) * 4;
    return max_n <= kSmallSort && bytes <= kSmallSortBytes ? (size_t)bytes : 0;
}
void launch_keys(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_keys, s.grid_p, s.tile, 0, st, a);
}
void launch_scan(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_scan, s.grid_c, kScanThreads, 0, st, a);
}
void launch_scatter(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_scatter, s.grid_p, s.tile, 0, st, a);
}
void launch_reorder(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_reorder, s.grid_p, s.tile, 0, st, a);
}
namespace {
// Traversal counters of one scene: [rows visited, candidates tested,
// in-range pairs (self included)], summed with int64 atomics.
__global__ void __launch_bounds__(256) k_traversal_stats(DevArrays a, int scene, unsigned long long* out) {
    const SceneDev& S = a.scenes[scene];
    unsigned long long rows = 0, cand = 0, hits = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.n; p += gridDim.x * blockDim.x) {
        const float4 xi = a.spos[S.p_off + p];
        const Probe q = probe_of(S, xi);
        const int R = S.reach;
        for (int dz = -R; dz <= R; ++dz)
            for (int dy = -R; dy <= R; ++dy) {
                const int z = q.c.cz + dz, y = q.c.cy + dy;
                int xl, xh;
                if (z < 0 || z >= S.nz || y < 0 || y >= S.ny || !row_span(S, q, y, z, &xl, &xh)) continue;
                const uint32_t row = row_key(a.tab, S, y, z);
                const uint32_t st = a.offsets[S.k_off + row + xl], en = a.offsets[S.k_off + row + xh + 1];
                ++rows;
                for (uint32_t j = st; j < en; ++j) {
                    const float4 xj = a.spos[S.p_off + j];
                    ++cand;
                    hits += dist2(fs(xi.x, xj.x), fs(xi.y, xj.y), fs(xi.z, xj.z)) <= S.smax;
                }
            }
    }
    for (int o = 16; o > 0; o >>= 1) {
        rows += __shfl_down_sync(kFull, rows, o);
        cand += __shfl_down_sync(kFull, cand, o);
        hits += __shfl_down_sync(kFull, hits, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, rows);
        atomicAdd(out + 1, cand);
        atomicAdd(out + 2, hits);
    }
}

__global__ void k_gather_by_id(const float4* __restrict__ pos, const float4* __restrict__ vel,
                               const float4* __restrict__ dyn, int p_off, int n, float* __restrict__ pos3,
                               float* __restrict__ vel3, float* __restrict__ dens, int32_t* __restrict__ sed) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const float4 x = pos[p_off + p];
    const int id = __float_as_int(x.w);
    if (id < 0 || id >= n) return;
    if (pos3) {
        pos3[3 * id] = x.x;
        pos3[3 * id + 1] = x.y;
        pos3[3 * id + 2] = x.z;
    }
    if (vel3 || sed) {
        const float4 v = vel[p_off + p];
        if (vel3) {
            vel3[3 * id] = v.x;
            vel3[3 * id + 1] = v.y;
            vel3[3 * id + 2] = v.z;
        }
        if (sed) sed[id] = __float_as_int(v.w);
    }
    if (dens) dens[id] = dyn[p_off + p].x;
}
}  // namespace

void launch_traversal_stats(const DevArrays& a, int scene, unsigned long long* out, cudaStream_t st) {
    k_traversal_stats<<<304, 256, 0, st>>>(a, scene, out);
}

// The readback's gather, one launch per scene, at the highest priority: its few
// blocks otherwise wait for every block of the neighbour pass that another
// system's stream has running, scene after scene.  Three systems of 39 scenes
// (216,000 particles) in turn, a pass of four steps and the readback, us: fast
// arithmetic 587 -> 508, exact 704 -> 584.
void launch_gather_by_id(const float4* pos, const float4* vel, const float4* dyn, int p_off, int n, float* pos3,
                         float* vel3, float* dens, int32_t* sed, int priority, cudaStream_t st) {
    if (n <= 0) return;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)((n + 255) / 256));
    c.blockDim = dim3(256);
    c.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributePriority;
    at.val.priority = priority;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, k_gather_by_id, pos, vel, dyn, p_off, n, pos3, vel3, dens, sed);
}

void configure_kernels() {
    const int bytes = kListCap * kMaxTile * (int)sizeof(uint32_t);
    cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSortBytes);
    cudaFuncSetAttribute(k_density<false, true, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_density<false, true, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_force<false, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_force<false, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

static size_t list_bytes(const LaunchShape& s) { return (size_t)kListCap * s.tile * sizeof(uint32_t); }

// Variant bit 2 relaxes the register budget of the two neighbour kernels
// (fewer resident blocks, no spills) against the default high occupancy.
// Bit 3 hands the in-range neighbour lists from the density pass to the force
// pass (takes precedence over bit 0) and ignores bit 2; bits 4 and 17 with it
// select the fast arithmetic of the force pass, bit 17 that of the density pass;
// bit 7 makes the packed 32-byte records part of the variant's memory.
// Variant bit 8 (with bit 3): the cooperative passes, G lanes per particle.
// Density: 32 lanes (bit 11: 16).  Force: 8 lanes (bit 9: 4, bit 10: 16).
// Bit 7 packs the force-pass inputs as in the per-lane passes; bit 2
// relaxes the force pass's register budget.
static void launch_density_coop(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    const bool pack = (s.variant & 128) != 0;
    if (s.variant & 2048) {
        if (pack)
            k_density_coop<16, true><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_density_coop<16, false><<<s.grid_p, s.tile, 0, st>>>(a);
    } else {
        if (pack)
            k_density_coop<32, true><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_density_coop<32, false><<<s.grid_p, s.tile, 0, st>>>(a);
    }
}

template <int MINB>
static void launch_force_coop_b(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    const bool pack = (s.variant & 128) != 0;
    const int gsel = (s.variant >> 9) & 3;
    if (gsel == 1) {
        if (pack)
            k_force_coop<4, true, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_force_coop<4, false, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
    } else if (gsel == 2) {
        if (pack)
            k_force_coop<16, true, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_force_coop<16, false, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
    } else {
        if (pack)
            k_force_coop<8, true, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_force_coop<8, false, MINB><<<s.grid_p, s.tile, 0, st>>>(a);
    }
}

// Bit 2 relaxes the cooperative force pass's register budget (3 resident
// blocks of 256 threads instead of 4).
static void launch_force_coop(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    if (s.variant & 4)
        launch_force_coop_b<3>(a, s, st);
    else
        launch_force_coop_b<4>(a, s, st);
}

static void launch_density_group(const DevArrays& a, const LaunchShape& s, bool fast, cudaStream_t st) {
    const int blocks = s.grid_p * s.tile / 8;
    // Blocks that wait for the one-block sort, the longest kernel of a small
    // step, hold most of the chip when they are more than two an SM, and other
    // systems' kernels out of it.  Three systems in turn, 64 captured steps, us,
    // early or not: 4,096 particles 855 vs 701, 2,500 604 vs 585, 1,500 527 vs
    // 526; one alone: 1,684 vs 1,683, 1,478 vs 1,486, 1,349 vs 1,380.  Launched
    // singly it pays at all of these (2,500 particles, 4 steps: 100 vs 112).
    const bool early = s.early && !(s.captured && s.sort_smem && blocks > 2 * s.nsm);
    const bool lane_lists = !s.force_group, pack = lane_lists && s.pack;
    if (fast)
        launch(early, k_density_group<true>, blocks, 256, 0, st, a, lane_lists, pack);
    else
        launch(early, k_density_group<false>, blocks, 256, 0, st, a, lane_lists, pack);
}

static void launch_force_group(const DevArrays& a, const LaunchShape& s, bool fast, cudaStream_t st) {
    const int blocks = s.grid_p * s.tile / 16;
    if (s.record) {
        if (fast)
            launch(s.early, k_force_group<true, true>, blocks, 256, 0, st, a);
        else
            launch(s.early, k_force_group<false, true>, blocks, 256, 0, st, a);
    } else if (fast)
        launch(s.early, k_force_group<true, false>, blocks, 256, 0, st, a);
    else
        launch(s.early, k_force_group<false, false>, blocks, 256, 0, st, a);
}

// Which passes of a step take a group of lanes per particle: the per-lane list
// forms (bit 8 without 256) of systems small enough to leave the chip idle with
// one lane per particle.  The lines are where the group passes stop paying
// when three systems run at once on streams of their own, which fills the chip
// first (us a step, group vs per lane; settled pools): exact arithmetic, both
// passes, 12,000 particles 26.8 vs 34.0, 16,000 32.4 vs 36.1, 20,000 40.6 vs
// 38.3; fast, density 8,000 19.7 vs 24.1, 12,000 24.5 vs 25.7, 16,000 29.0 vs
// 27.1; fast, force (beside the group density pass) 8,000 19.1 vs 19.7, 12,000
// 26.5 vs 24.5.  A system alone on the chip gains up to there from 2.3x (1,000
// particles: 74 to 32 us) to 1.6x (20,000: 99 to 62 us) a step (all of this
// with the sort in four kernels).
// The ordered passes' line: density + force, us, a warp per particle vs one lane,
// 5,000 particles 34 vs 127, 16,384 68 vs 143, 50,000 167 vs 217, 200,000 607 vs
// 536.
void group_rules(LaunchShape& s) {
    const int64_t n = (int64_t)s.grid_p * s.tile;
    const bool lists = (s.variant & (8 | 256)) == 8;
    s.early = n <= 18432;
    s.ordered_group = n <= 32768;
    s.density_group = lists && n <= ((s.variant & 131072) ? 12288 : 18432);
    s.force_group = s.density_group && n <= ((s.variant & (131072 | 16)) == (131072 | 16) ? 8192 : 18432);
}

static bool coop(const LaunchShape& s) { return (s.variant & (256 | 8)) == (256 | 8); }

// The bits that the launchers below act on, by the form that they take.
int neighbour_kernels(const LaunchShape& s) {
    if (coop(s)) return s.variant;
    if (!(s.variant & 8)) return s.variant & (1 | 4);
    const bool tma = s.fmap && (s.variant & 128) && !s.force_group;
    return (s.variant & (8 | 16 | 131072 | (tma ? 262144 : 0))) | (s.pack ? 128 : 0);
}

void launch_density(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    if (coop(s)) {
        launch_density_coop(a, s, st);
        return;
    }
    const bool relaxed = (s.variant & 4) != 0;
    if (s.density_group) {
        launch_density_group(a, s, (s.variant & 131072) != 0, st);
    } else if (s.variant & 8) {
        if (s.variant & 131072)
            k_density_list<true><<<s.grid_p, s.tile, (size_t)s.tile * kBuf * 4, st>>>(a, s.pack);
        else
            k_density_list<false><<<s.grid_p, s.tile, (size_t)s.tile * kBuf * 4, st>>>(a, s.pack);
    } else if (s.variant & 1) {
        if (relaxed)
            k_density<false, true, 4><<<s.grid_p, s.tile, list_bytes(s), st>>>(a);
        else
            k_density<false, true, 8><<<s.grid_p, s.tile, list_bytes(s), st>>>(a);
    } else {
        if (relaxed)
            k_density<false, false, 4><<<s.grid_p, s.tile, 0, st>>>(a);
        else
            k_density<false, false, 8><<<s.grid_p, s.tile, 0, st>>>(a);
    }
}
void launch_density_ordered(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    if (s.ordered_group)
        launch(s.early, k_density_ordered, s.grid_p * s.tile / 8, 256, 0, st, a);
    else
        k_density<true, false, 1><<<s.grid_p, s.tile, 0, st>>>(a);
}
void launch_force(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    if (coop(s)) {
        launch_force_coop(a, s, st);
        return;
    }
    if (s.force_group) {
        launch_force_group(a, s, (s.variant & (131072 | 16)) == (131072 | 16), st);
        return;
    }
    // The list variants walk their lists (or, on overflow, the cells) per
    // lane: over the packed records wherever the system holds them, since that
    // form is the fastest at every size measured; warps take their work in
    // slices from a counter.
    if ((s.variant & 262144) && (s.variant & (131072 | 128 | 24)) == (131072 | 128 | 24) && s.fmap) {
        // bit 18: the TMA gather pipeline (fast arithmetic, packed records)
        k_force_tma<3><<<s.grid_p, s.tile + 32, force_tma_smem(s.tile), st>>>(a, *static_cast<const CUtensorMap*>(s.fmap));
        return;
    }
    if (s.variant & 8) {
        const bool fast = (s.variant & (131072 | 16)) == (131072 | 16);
        if (!s.pack) {
            if (fast)
                k_force<false, 4, true, true, true><<<s.grid_dyn, s.tile, 0, st>>>(a);
            else
                k_force<false, 4, true, true><<<s.grid_dyn, s.tile, 0, st>>>(a);
        } else if (s.record) {
            if (fast)
                k_force_rec<true, true><<<s.grid_dyn, s.tile, 0, st>>>(a);
            else
                k_force_rec<false, true><<<s.grid_dyn, s.tile, 0, st>>>(a);
        } else if (fast)
            k_force_rec<true, false><<<s.grid_dyn, s.tile, 0, st>>>(a);
        else
            k_force_rec<false, false><<<s.grid_dyn, s.tile, 0, st>>>(a);
    } else if (s.variant & 4)
        k_force<false, 3><<<s.grid_p, s.tile, list_bytes(s), st>>>(a);
    else
        k_force<false, 4><<<s.grid_p, s.tile, list_bytes(s), st>>>(a);
}
void launch_force_ordered(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    if (s.ordered_group)
        launch(s.early, k_force_ordered, s.grid_p * s.tile / 8, 256, 0, st, a);
    else
        k_force<true, 1><<<s.grid_p, s.tile, 0, st>>>(a);
}
void launch_terrain(const DevArrays& a, const LaunchShape& s, cudaStream_t st) {
    launch(s.early, k_terrain, (s.grid_t * (s.tile / 4) + 255) / 256, 256, 0, st, a);
}
void launch_tick(const DevArrays& a, const LaunchShape& s, int nscenes, cudaStream_t st) {
    launch(s.early, k_tick, (nscenes + 127) / 128, 128, 0, st, a.steps_left, nscenes, s.early);
}
void launch_neighbour_counts(const DevArrays& a, const LaunchShape& s, int32_t* out_by_id, cudaStream_t st) {
    k_neighbour_counts<<<s.grid_p, s.tile, 0, st>>>(a, out_by_id);
}
void launch_diag(const DevArrays& a, int nlist, double* partial, long long* isums, int* nan_count,
                 cudaStream_t st) {
    if (nlist > 0) k_diag<<<nlist * kDiagBlocks, 256, 0, st>>>(a, partial, isums, nan_count);
}

}  // namespace sph
