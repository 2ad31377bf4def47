// The ALE remap step on sm_100a: ale_remap_step (ale_remap/ale_remap.F90:76-188)
// in two kernels over tiles of columns staged in shared memory.
//
//   k_ale_columns  a block per tile of adjacent cell columns: the column total
//                  (L1), h_ref (L2), the h_old snapshot (L3), the zstar
//                  targets (L4, :478-527) and the commit (L9 mass budget,
//                  h_layer = target_h, L10 bt_eta); every tracer of the launch
//                  remapped over the tile's geometry (L5/L6,
//                  ocean_remap_tracer_field :530-581, heat / salt budgets).
//   k_ale_faces    a block per tile of u faces or v faces: face thicknesses
//                  from the two adjacent cells, remap of the velocity, optional
//                  KE-conserving rescale (L7/L8, :584-724).
//
// The column remap is remap_column (ale_remap/kernel_remap.F90:43-376) for PCM,
// PLM and PPM. The reference sweeps each column serially: for new layer k it
// walks the old layers from a start index carried over from layer k-1 and sums
// the pieces whose overlap is positive. When every old and new thickness of a
// column is >= 0 both sets of interface depths are non-decreasing, and the old
// layers with positive overlap with new layer k are exactly those in the
// contiguous range [first old layer whose bottom lies below z_new(k-1), last old
// layer whose top lies above z_new(k)]; summed in increasing order they give
// the reference's integral bit for bit. So each (column, layer) is computed by
// its own thread from the tile, in passes that every lane of a warp takes alike:
//
//   geometry  once per tile, for all its tracers: the interface depths (one
//             thread per column, the reference's running sums), then per new
//             interface the old layer that holds it and its position xi in that
//             layer, and per old layer the position xf of its own bottom. A
//             piece of the reference is bounded by new interfaces (xi) and old
//             ones (0 or xf), so these are every quotient its pieces form.
//   layers    per tracer and old layer: the limited PPM parabola (PLM: slope).
//   pieces    per tracer and new layer: the pieces between its two interfaces.
//
// A column with a negative or NaN thickness takes the reference's serial sweep
// instead, on one thread, from the same tile. The column total is the last old
// interface depth: the same additions in the same order.
// What bounds both kernels is instruction issue and the latency of FP64 chains at
// 23 and 30 warps per SM (shared memory holds whole columns), not bytes: 790 and
// 900 thread instructions per (column, layer) of two fields, issued in 47 and 67 %
// of the cycles, against about 2000 with one thread per (column, new layer) that
// searched, divided and evaluated the parabola anew for every piece and field. k_ale_columns (T, S) and
// k_ale_faces at 479x303x30: 404 -> 222 us and 355 -> 181 us; at 1444x1084x75:
// 19.2 -> 6.8 ms and 16.6 -> 6.1 ms (0.30 and 0.14 of the bytes' time at 6537 GB/s).
// Compiled with -fmad=false: results are the reference's IEEE sequence.

#include <cuda_runtime.h>

#include <climits>
#include <cstdio>
#include <string>

#include "ale_b200.h"
#include "redi_kernels.h"

namespace {

constexpr double kHFloor = 1.5e-4;  // ale_remap/ale_remap.F90:70 H_FLOOR
constexpr int kNzMax = ALE_B200_NZ_MAX;
constexpr int kThreadsMax = 256;
constexpr int kMaxTracers = 8;  // tracers remapped by one launch
constexpr int kPCM = 1, kPLM = 2, kPPM = 3;

thread_local std::string g_err;

struct Dims {
    int nx, ny, nz;
    int n2;  // cells per layer (every offset of a step fits in 32 bits: checked on the host)
};

struct TracerSet {
    int n;
    double* tr[kMaxTracers];
    double* budget[kMaxTracers];
};

// A column of a tile in shared memory: element k at p[k * S].
template <int S>
struct Col {
    const double* p;
    __device__ __forceinline__ double operator[](int k) const { return p[k * S]; }
};

// PLM slope of old layer ko (1-based), kernel_remap.F90:163-174
template <class A>
__device__ __forceinline__ double plm_slope(const A& q, int nz, int ko) {
    if (ko == 1 || ko == nz) return 0.0;
    const double dq_l = q[ko - 1] - q[ko - 2];
    const double dq_r = q[ko] - q[ko - 1];
    if (dq_l * dq_r > 0.0) return 0.5 * copysign(fmin(fabs(dq_l), fabs(dq_r)), dq_l);
    return 0.0;
}

// Limited PPM edges and curvature of old layer ko (1-based), nz >= 3:
// kernel_remap.F90:257-328 evaluated for one layer.
template <class A>
__device__ __forceinline__ void ppm_coeffs(const A& q, int nz, int ko, double& qL, double& qR, double& q6) {
    const double qc = q[ko - 1];
    double l, r;
    if (ko == 1) {
        l = qc;
    } else if (ko == 2) {
        l = 0.5 * (q[0] + q[1]);  // q_L(2) = q_R(1)
    } else {                      // the interior edge between layers ko-1 and ko
        const int k = ko - 1;
        l = 0.5 * (q[k - 1] + q[k]);
        if (k + 2 <= nz) l = (7.0 / 12.0) * (q[k - 1] + q[k]) - (1.0 / 12.0) * (q[k - 2] + q[k + 1]);
    }
    if (ko == nz) {
        r = qc;
    } else if (ko == 1) {
        r = 0.5 * (q[0] + q[1]);
    } else {  // the interior edge between layers ko and ko+1
        const int k = ko;
        r = 0.5 * (q[k - 1] + q[k]);
        if (k + 2 <= nz) r = (7.0 / 12.0) * (q[k - 1] + q[k]) - (1.0 / 12.0) * (q[k - 2] + q[k + 1]);
    }
    double q_min = qc, q_max = qc;
    if (ko > 1) {
        q_min = fmin(q_min, q[ko - 2]);
        q_max = fmax(q_max, q[ko - 2]);
    }
    if (ko < nz) {
        q_min = fmin(q_min, q[ko]);
        q_max = fmax(q_max, q[ko]);
    }
    l = fmax(q_min, fmin(q_max, l));
    r = fmax(q_min, fmin(q_max, r));
    const double dq = r - l;
    const double dq_l = qc - l;
    const double dq_r = r - qc;
    if (dq_l * dq_r <= 0.0) {
        l = qc;
        r = qc;
    } else {
        const double s6 = 6.0 * qc - 3.0 * (l + r);
        if (fabs(s6) > fabs(dq)) {
            if (s6 * dq > 0.0)
                l = 3.0 * qc - 2.0 * r;
            else
                r = 3.0 * qc - 2.0 * l;
        }
    }
    qL = l;
    qR = r;
    q6 = 6.0 * qc - 3.0 * (l + r);
}

// Old layer ko's contribution to a new layer: the integral of its
// reconstruction over [z_lo, z_hi] (kernel_remap.F90:107, 193-204, 349-362).
template <int M, class A>
__device__ __forceinline__ double piece(const A& q, const A& dz_old, int nz, int ko, double zo_lo, double z_lo,
                                        double z_hi, double overlap) {
    const double qo = q[ko - 1];
    if (M == kPCM) return qo * overlap;
    const double d = dz_old[ko - 1];
    if (!(d > 0.0)) return qo * overlap;
    const double xi_lo = (z_lo - zo_lo) / d;
    const double xi_hi = (z_hi - zo_lo) / d;
    if (M == kPLM) return overlap * (qo + plm_slope(q, nz, ko) * (xi_lo + xi_hi - 1.0));
    double cL, cR, c6;
    ppm_coeffs(q, nz, ko, cL, cR, c6);
    return d * ((xi_hi - xi_lo) * cL + 0.5 * (xi_hi * xi_hi - xi_lo * xi_lo) * (cR - cL + c6) -
                (xi_hi * xi_hi * xi_hi - xi_lo * xi_lo * xi_lo) * c6 / 3.0);
}

// The reference's serial sweep (remap_column), for columns with a negative or NaN
// thickness or with averages that are not finite. The old interface depths are
// the running sums of dz_old, formed as they are needed. Latency of one thread a
// column and field: the tracers of a launch are swept side by side (300x250x30, every
// column with a negative layer, 3 tracers: 1.64 ms, one after another 2.17).
template <int METHOD, class A, class Dz, class Emit>
__device__ __noinline__ void serial_column(int nz, const A dz_old, const Dz dz_new, const A q, const Emit emit) {
    if (METHOD != kPCM && nz == 1) {
        emit(0, q[0]);
        return;
    }
    int ko_start = 1;
    double zn_prev = 0.0, z_start = 0.0;  // z_start: top of old layer ko_start
    for (int k = 1; k <= nz; ++k) {
        const double dzn = dz_new(k - 1);
        const double zn = zn_prev + dzn;
        if (dzn <= 0.0) {
            emit(k - 1, 0.0);
            zn_prev = zn;
            continue;
        }
        double integral = 0.0;
        double zo_hi = z_start;
        for (int ko = ko_start; ko <= nz; ++ko) {
            const double zo_lo = zo_hi;
            zo_hi = zo_lo + dz_old[ko - 1];
            const double z_lo = fmax(zn_prev, zo_lo);
            const double z_hi = fmin(zn, zo_hi);
            const double overlap = z_hi - z_lo;
            if (overlap <= 0.0) {
                if (zo_hi > zn) break;
                continue;
            }
            integral = integral + piece<METHOD>(q, dz_old, nz, ko, zo_lo, z_lo, z_hi, overlap);
            if (zo_hi <= zn) {
                ko_start = ko;
                z_start = zo_lo;
            }
        }
        emit(k - 1, integral / dzn);
        zn_prev = zn;
    }
}

// x / 3 as the correctly rounded quotient (the reference divides): the product
// with the rounded reciprocal is within one ulp, the fused remainder is exact,
// and the corrected quotient is the rounded one (Markstein, IBM J. Res. Dev.
// 34, 1990). Three FP64 operations instead of a general division; infinities
// pass through.
__device__ __forceinline__ double third(double x) {
    constexpr double y = 1.0 / 3.0;
    const double q = x * y;
    const double r = __fma_rn(-3.0, q, x);
    const double t = __fma_rn(r, y, q);
    return fabs(x) <= 1.7976931348623157e308 ? t : x;
}

__device__ __forceinline__ bool finite(double x) { return fabs(x) <= 1.7976931348623157e308; }
// fmin(a, x) and fmax(a, x) for a that is not NaN (the sign of a zero apart,
// which no result keeps): one compare and a select.
__device__ __forceinline__ double lesser(double a, double x) { return x < a ? x : a; }
__device__ __forceinline__ double greater(double a, double x) { return x > a ? x : a; }

// Arrays of a tile with nt fields and `extra` more: five of geometry, and per
// field the averages (PPM: then the left edges) and, PLM, the slopes or, PPM, two
// more coefficients, the first field's in the place of the interface depths.
__host__ __device__ constexpr int tile_arrays(int method, int nt, int extra) {
    return extra + (method == kPPM ? 5 + nt + 2 * (nt - 1) : 5 + 2 * nt);
}
// Shared memory of one column of a tile: its arrays and its layer indices.
constexpr size_t column_bytes(int nz, int arrays) { return (size_t)(nz + 1) * (8 * arrays + 1); }

// A tile of W columns in shared memory with NT fields remapped together: nz + 1
// rows, row k holding kArrays values of every column side by side, so that one
// index and compile-time offsets reach everything a thread reads around layer
// k, and the lanes of a warp (neighbouring columns) touch neighbouring words.
// The interface depths are dead once the positions are known, and the averages
// once the parabolas are; a PPM launch keeps the parabolas in their place.
// ko, per new interface k: the old layer that holds it (0-based); bit 7: new
// layer k overlaps no old layer.
template <int METHOD, int W, int NT, int EXTRA>
struct Tile {
    static constexpr int D = 0;   // old thicknesses
    static constexpr int XI = 1;  // per new interface: its position in the old layer that holds it
    static constexpr int XF = 2;  // per old layer: the position of its bottom
    static constexpr int ZO = 3, ZN = 4;  // old and new interface depths
    static constexpr int S = tile_arrays(METHOD, NT, EXTRA) * W;  // row stride
    static __device__ constexpr int Q(int n) { return 5 + n; }             // layer averages
    static __device__ constexpr int L(int n) { return METHOD == kPPM ? Q(n) : 5 + NT + n; }  // left edge; PLM: slope
    static __device__ constexpr int B(int n) { return n == 0 ? ZN : 5 + NT + 2 * (n - 1); }  // PPM: cR - cL + c6
    static __device__ constexpr int C6(int n) { return n == 0 ? ZO : 6 + NT + 2 * (n - 1); }

    double* p;          // this thread's column
    unsigned char* ko;  // its layer indices, W apart
    __device__ __forceinline__ Tile(double* sm, int nz, int c)
        : p(sm + c), ko(reinterpret_cast<unsigned char*>(sm + (nz + 1) * S) + c) {}
    __device__ __forceinline__ double& at(int array, int k) const { return p[k * S + array * W]; }
    __device__ __forceinline__ Col<S> col(int array) const { return Col<S>{p + array * W}; }
};

// New interfaces [ka, kb): for each the first old layer whose bottom lies below
// it (the last layer if none does), its position there, and whether the new
// layer below it overlaps no old layer; the positions of the bottoms of old
// layers [ka, kb). Vanished layers get position 0, so they never contribute.
template <class T>
__device__ __forceinline__ void tile_positions(const T& t, int nz, int W, int ka, int kb) {
    if (ka >= kb) return;
    double z = t.at(T::ZN, ka);
    int lo = 1, hi = nz;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (t.at(T::ZO, mid) > z)
            hi = mid;
        else
            lo = mid + 1;
    }
    const double bed = t.at(T::ZO, nz);
    double zo_hi = t.at(T::ZO, lo);
    for (int k = ka; k < kb; ++k) {
        while (lo < nz && !(zo_hi > z)) zo_hi = t.at(T::ZO, ++lo);
        const double zo_lo = t.at(T::ZO, lo - 1);
        const double dl = t.at(T::D, lo - 1);
        t.at(T::XI, k) = dl > 0.0 ? (fmin(z, zo_hi) - zo_lo) / dl : 0.0;
        int flag = lo - 1;  // nz <= 128: bit 7 is free
        if (k < nz) {
            const double z_next = t.at(T::ZN, k + 1);
            if (!(fmin(z_next, bed) > z)) flag |= 0x80;
            const double dk = t.at(T::D, k);
            t.at(T::XF, k) = dk > 0.0 ? (t.at(T::ZO, k + 1) - t.at(T::ZO, k)) / dk : 0.0;
            z = z_next;
        }
        t.ko[k * W] = (unsigned char)flag;
    }
}

// PLM slopes of old layers [ka, kb) of field n.
template <class T>
__device__ __forceinline__ void tile_slopes(const T& t, int n, int nz, int ka, int kb) {
    for (int k = ka; k < kb; ++k) t.at(T::L(n), k) = plm_slope(t.col(T::Q(n)), nz, k + 1);
}

// The averages around old layers [ka, kb) of a field that other threads own.
struct Halo {
    double m2, m1, p1, p2;  // layers ka - 2, ka - 1, kb, kb + 1 (clamped to the column)
};
template <class T>
__device__ __forceinline__ Halo tile_halo(const T& t, int n, int nz, int ka, int kb) {
    const int Q = T::Q(n);
    return Halo{t.at(Q, max(ka - 2, 0)), t.at(Q, min(max(ka - 1, 0), nz - 1)), t.at(Q, min(kb, nz - 1)),
                t.at(Q, min(kb + 1, nz - 1))};
}

// The limited PPM parabolas (kernel_remap.F90:257-328) of old layers [ka, kb) of
// field n from finite averages, which the left edges replace. The edge between
// two layers and the smaller and larger of their averages serve both.
template <class T>
__device__ __forceinline__ void tile_parabolas(const T& t, int n, const Halo h, int nz, int ka, int kb) {
    if (ka >= kb) return;
    const int Q = T::Q(n);
    double qc = t.at(Q, ka);
    double qm = ka > 0 ? h.m1 : qc, qp = ka + 1 < kb ? t.at(Q, ka + 1) : h.p1;
    // the raw edge between layers k and k+1
    auto edge = [nz](int k, double q0, double q1, double q2, double q3) {
        return k == 0 || k == nz - 2 ? 0.5 * (q1 + q2) : (7.0 / 12.0) * (q1 + q2) - (1.0 / 12.0) * (q0 + q3);
    };
    double left = ka == 0 ? qc : edge(ka - 1, h.m2, qm, qc, qp);
    double lo = lesser(qm, qc), hi = greater(qm, qc);
    for (int k = ka; k < kb; ++k) {
        const double qn = k + 2 < kb ? t.at(Q, k + 2) : k + 2 == kb ? h.p1 : h.p2;
        const double right = k == nz - 1 ? qc : edge(k, qm, qc, qp, qn);
        const double lo1 = lesser(qc, qp), hi1 = greater(qc, qp);
        const double q_min = lesser(lo, lo1), q_max = greater(hi, hi1);
        double l = greater(q_min, lesser(q_max, left)), r = greater(q_min, lesser(q_max, right));
        const double q6 = 6.0 * qc, q3 = 3.0 * qc;
        const double dq = r - l, dq_l = qc - l, dq_r = r - qc;
        const double s6 = q6 - 3.0 * (l + r);
        const bool flat = dq_l * dq_r <= 0.0, over = fabs(s6) > fabs(dq), pos = s6 * dq > 0.0;
        const double l2 = q3 - 2.0 * r, r2 = q3 - 2.0 * l;
        if (over && pos) l = l2;
        if (over && !pos) r = r2;
        if (flat) l = r = qc;
        const double c6 = q6 - 3.0 * (l + r);
        t.at(T::L(n), k) = l;
        t.at(T::B(n), k) = r - l + c6;
        t.at(T::C6(n), k) = c6;
        qm = qc;
        qc = qp;
        qp = qn;
        left = right;
        lo = lo1;
        hi = hi1;
    }
}

// New layers [ka, kb): the integral of each field over each, from the pieces of
// the old layers between its two interfaces; emit(k, integrals, what fetch(k)
// gave: fetched one layer ahead). A thread walks its layers downwards: the old
// layer that holds an interface is the last of one new layer and the first of
// the next, and its coefficients stay in registers.
template <int METHOD, int NT, class T, class Fetch, class Emit>
__device__ __forceinline__ void tile_integrals(const T& t, int W, int ka, int kb, Fetch fetch, Emit emit) {
    if (ka >= kb) return;
    auto next = fetch(ka);
    double d0, l0[NT], b0[NT], c0[NT];  // old layer p0
    auto load = [&](int p) {
        d0 = t.at(T::D, p);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (METHOD == kPPM) {
                l0[n] = t.at(T::L(n), p);
                b0[n] = t.at(T::B(n), p);
                c0[n] = t.at(T::C6(n), p);
            } else {
                b0[n] = t.at(T::Q(n), p);
                if (METHOD == kPLM) l0[n] = t.at(T::L(n), p);
            }
        }
    };
    int f = t.ko[ka * W], p0 = f & 0x7f;
    double x0 = t.at(T::XI, ka);
    load(p0);
    for (int k = ka; k < kb; ++k) {
        const int f1 = t.ko[(k + 1) * W], p1 = f1 & 0x7f;
        const double x1 = t.at(T::XI, k + 1);
        const auto got = next;
        if (k + 1 < kb) next = fetch(k + 1);
        double sum[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) sum[n] = 0.0;
        // the piece of the loaded layer between positions xl and xh (PLM, PCM: depths zl and zh)
        auto add = [&](double xl, double xh, double zl, double zh) {
            if (METHOD == kPPM) {
                const double a1 = xh - xl, a2 = 0.5 * (xh * xh - xl * xl), a3 = xh * xh * xh - xl * xl * xl;
#pragma unroll
                for (int n = 0; n < NT; ++n) sum[n] = sum[n] + d0 * (a1 * l0[n] + a2 * b0[n] - third(a3 * c0[n]));
            } else {
                const double overlap = zh - zl;
#pragma unroll
                for (int n = 0; n < NT; ++n)
                    sum[n] = sum[n] + (METHOD == kPLM ? overlap * (b0[n] + l0[n] * (xl + xh - 1.0)) : b0[n] * overlap);
            }
        };
        auto z = [&](int array, int row) { return METHOD == kPPM ? 0.0 : t.at(array, row); };
        const bool some = !(f & 0x80), inside = p1 == p0;
        if (some)
            add(x0, inside ? x1 : t.at(T::XF, p0), z(T::ZN, k),
                inside ? fmin(z(T::ZN, k + 1), z(T::ZO, p0 + 1)) : z(T::ZO, p0 + 1));
        if (!inside) {
            if (some) {
                for (int p = p0 + 1; p < p1; ++p) {
                    const double xf = t.at(T::XF, p);
                    if (xf <= 0.0) continue;
                    load(p);
                    add(0.0, xf, z(T::ZO, p), z(T::ZO, p + 1));
                }
            }
            load(p1);
            if (some && !(x1 <= 0.0)) add(0.0, x1, z(T::ZO, p1), fmin(z(T::ZN, k + 1), z(T::ZO, p1 + 1)));
        }
        emit(k, sum, got);
        f = f1;
        p0 = p1;
        x0 = x1;
    }
}

// rescale_anomaly_ke (ale_remap/ale_remap.F90:684-724) on one column: u_old(k)
// is read, u_new[k * S] updated in place.
template <int S, class U>
__device__ void rescale_anomaly_ke(int nz, const Col<S> h_old, const Col<S> h_new, const U u_old, double* u_new) {
    double h_old_sum = 0.0, h_new_sum = 0.0, mom_old = 0.0, mom_new = 0.0;
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        h_old_sum = h_old_sum + h_old[k];
        h_new_sum = h_new_sum + h_new[k];
        mom_old = mom_old + h_old[k] * u_old(k);
        mom_new = mom_new + h_new[k] * u_new[k * S];
    }
    if (h_old_sum <= kHFloor || h_new_sum <= kHFloor) return;
    const double u_bar_old = mom_old / h_old_sum;
    const double u_bar_new = mom_new / h_new_sum;
    double ke_old = 0.0, ke_new = 0.0;
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        double anom = u_old(k) - u_bar_old;
        ke_old = ke_old + 0.5 * h_old[k] * anom * anom;
        anom = u_new[k * S] - u_bar_new;
        ke_new = ke_new + 0.5 * h_new[k] * anom * anom;
    }
    if (ke_new <= 0.0 || ke_old <= 0.0) return;
    double scale_fac = sqrt(ke_old / ke_new);
    if (scale_fac > 1.25) scale_fac = 1.25;
    if (scale_fac < 0.0) scale_fac = 0.0;
    for (int k = 0; k < nz; ++k) u_new[k * S] = u_bar_new + scale_fac * (u_new[k * S] - u_bar_new);
}

// ----------------------------------------------------------------- kernels --
// A block is W columns times G = blockDim.x / W rows of threads; row r of
// threads works on the contiguous layers [ka, kb) of its column.
struct Rows {
    int ka, kb;
    __device__ __forceinline__ Rows(int nz, int G, int r) {
        const int n = (nz + G - 1) / G;
        ka = min(r * n, nz);
        kb = min(ka + n, nz);
    }
};

// Tile of cell columns. first: the first launch of a step (writes the snapshot,
// the targets, total_h and h_ref); commit: the last one (mass budget, h_layer,
// bt_eta). h_layer and bt_eta keep the old state until the commit, so every
// launch forms the same targets from them.
template <int METHOD, int W, int NT>
__global__ void __launch_bounds__(kThreadsMax, 3) k_ale_columns(
    const Dims d, const TracerSet ts, int first, int commit, double* h_layer, double* bt_eta,
    const double* __restrict__ bt_H_ref, const double* __restrict__ dsig, double* total_h, double* h_ref, double* h_old,
    double* target_h, double* mass_budget) {
    using T = Tile<METHOD, W, NT, 0>;
    static_assert(NT <= 2, "a block has at least two rows of threads");
    extern __shared__ double sm[];
    __shared__ int serial[W];
    __shared__ double ct[W];  // column total h_ref + eta of the zstar target
    const int nz = d.nz;
    const int n2 = d.n2;
    const int c = threadIdx.x % W, r = threadIdx.x / W;
    const T t(sm, nz, c);
    const Rows rows(nz, blockDim.x / W, r);
    const int ka = rows.ka, kb = rows.kb;
    const int col = blockIdx.x * W + c;
    const bool in = col < n2;

    // Global loads are issued in batches of kBatch layers ahead of the stores that
    // follow them (the arrays are updated in place, so the compiler cannot).
    constexpr int kBatch = 4;
    // the averages of tracers n0 .. n0 + NT - 1 (a slot beyond the last repeats it and is not written)
    auto stage = [&](int n0) {
        bool ok = true;
        const double* tr[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) tr[n] = ts.tr[min(n0 + n, ts.n - 1)] + col;
        for (int k0 = ka; k0 < kb; k0 += kBatch) {
            double x[NT][kBatch];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < kBatch; ++i) x[n][i] = tr[n][n2 * min(k0 + i, kb - 1)];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (k0 + i >= kb) break;
                const double h = t.at(T::D, k0 + i);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const double q = h > kHFloor ? x[n][i] / h : 0.0;
                    ok = ok && finite(q);
                    t.at(T::Q(n), k0 + i) = q;
                }
            }
        }
        if (!ok) serial[c] = 1;
    };

    if (in) {
        for (int k0 = ka; k0 < kb; k0 += kBatch) {
            double h[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) h[i] = h_layer[col + n2 * min(k0 + i, kb - 1)];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (k0 + i >= kb) break;
                t.at(T::D, k0 + i) = h[i];
                if (first) h_old[col + n2 * (k0 + i)] = h[i];  // L3
            }
        }
        if (r == 0) serial[c] = 0;
    }
    __syncthreads();
    if (in && r == 0) {
        // L1 total (the running sum of the column: the last interface depth), L2 h_ref, L4 column total, L10
        double s = 0.0;
        bool mono = true;
        t.at(T::ZO, 0) = 0.0;
#pragma unroll 4
        for (int k = 0; k < nz; ++k) {
            const double x = t.at(T::D, k);
            mono = mono && x >= 0.0;
            s = s + x;
            t.at(T::ZO, k + 1) = s;
        }
        const double e = bt_eta[col];
        const double hr = s - e;
        if (first) {
            if (total_h) total_h[col] = s;
            if (h_ref) h_ref[col] = hr;
        }
        const double tot = hr + e;
        ct[c] = tot;
        double z = 0.0, eta = -__ldg(bt_H_ref + col);
        t.at(T::ZN, 0) = 0.0;
#pragma unroll 4
        for (int k = 0; k < nz; ++k) {
            const double y = tot * __ldg(dsig + k);
            mono = mono && y >= 0.0;
            z = z + y;
            eta = eta + y;
            t.at(T::ZN, k + 1) = z;
        }
        if (commit) bt_eta[col] = eta;
        if (!mono) serial[c] = 1;
    }
    if (in && ts.n > 0) stage(0);  // the other rows of threads wait for their loads meanwhile
    __syncthreads();
    const double tot = in ? ct[c] : 0.0;
    if (in) {
        if (first || commit) {  // L4 targets, L9
            for (int k0 = ka; k0 < kb; k0 += kBatch) {
                double m[kBatch];
                if (commit) {
#pragma unroll
                    for (int i = 0; i < kBatch; ++i) m[i] = mass_budget[col + n2 * min(k0 + i, kb - 1)];
                }
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int k = k0 + i, o = col + n2 * k;
                    if (k >= kb) break;
                    const double tg = tot * __ldg(dsig + k);
                    if (first) target_h[o] = tg;
                    if (commit) {
                        mass_budget[o] = m[i] + (tg - t.at(T::D, k));
                        h_layer[o] = tg;
                    }
                }
            }
        }
        if (!serial[c]) tile_positions(t, nz, W, ka, kb == nz && ka < kb ? nz + 1 : kb);
    }
    for (int n0 = 0; n0 < ts.n; n0 += NT) {
        if (n0 > 0 && in) stage(n0);
        __syncthreads();
        const bool ser = in && serial[c];
        if (METHOD == kPPM) {
            Halo h[NT];
            if (in && !ser) {
#pragma unroll
                for (int n = 0; n < NT; ++n) h[n] = tile_halo(t, n, nz, ka, kb);
            }
            __syncthreads();
            if (in && !ser) {
#pragma unroll
                for (int n = 0; n < NT; ++n) tile_parabolas(t, n, h[n], nz, ka, kb);
            }
            __syncthreads();
        } else if (METHOD == kPLM) {
            if (in && !ser) {
#pragma unroll
                for (int n = 0; n < NT; ++n) tile_slopes(t, n, nz, ka, kb);
            }
            __syncthreads();
        }
        if (in && !ser) {
            double *tr[NT], *budget[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int m = min(n0 + n, ts.n - 1);
                tr[n] = ts.tr[m] + col;
                budget[n] = ts.budget[m] ? ts.budget[m] + col : nullptr;
            }
            struct Old {
                double tr[NT], budget[NT];
            };
            tile_integrals<METHOD, NT>(
                t, W, ka, kb,
                [&](int k) {
                    Old o;
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        o.tr[n] = budget[n] ? tr[n][n2 * k] : 0.0;
                        o.budget[n] = budget[n] ? budget[n][n2 * k] : 0.0;
                    }
                    return o;
                },
                [&](int k, const double(&sum)[NT], const Old& old) {
                    const double dzn = tot * __ldg(dsig + k);
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (n0 + n >= ts.n) break;
                        double cn = dzn <= 0.0 ? 0.0 : sum[n] / dzn;
                        if (METHOD != kPCM && nz == 1) cn = t.at(T::Q(n), 0);
                        const double hTr_new = cn * dzn;
                        if (budget[n]) budget[n][n2 * k] = old.budget[n] + (hTr_new - old.tr[n]);
                        tr[n][n2 * k] = hTr_new;
                    }
                });
        } else if (ser && r < NT && n0 + r < ts.n) {  // a tracer on each of the first rows of threads
            double* tr = ts.tr[n0 + r] + col;
            double* b = ts.budget[n0 + r] ? ts.budget[n0 + r] + col : nullptr;
            serial_column<METHOD>(
                nz, t.col(T::D), [=](int k) { return tot * __ldg(dsig + k); }, t.col(T::Q(r)),
                [=](int k, double cn) {
                    const double hTr_new = cn * (tot * __ldg(dsig + k));
                    if (b) b[n2 * k] = b[n2 * k] + (hTr_new - tr[n2 * k]);
                    tr[n2 * k] = hTr_new;
                });
        }
        __syncthreads();  // the tracer arrays are reused by the next tracers
    }
}

// Tile of u faces (blocks [0, nbu)) or v faces (the rest). KE: the KE-conserving
// rescale, which needs the column's new values together.
template <int METHOD, int W, bool KE>
__global__ void __launch_bounds__(kThreadsMax, 4) k_ale_faces(const Dims d, int nbu, const double* __restrict__ h_old,
                                                              const double* __restrict__ target_h, double* u,
                                                              double* v) {
    using T = Tile<METHOD, W, 1, KE ? 2 : 1>;
    constexpr int DZ = tile_arrays(METHOD, 1, 0), QN = DZ + (KE ? 1 : 0);  // new thicknesses; new values
    extern __shared__ double sm[];
    __shared__ int serial[W];
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int n2 = d.n2;
    const int c = threadIdx.x % W, r = threadIdx.x / W;
    const T t(sm, nz, c);
    const Rows rows(nz, blockDim.x / W, r);
    const int ka = rows.ka, kb = rows.kb;
    const bool xface = (int)blockIdx.x < nbu;
    const int nf = xface ? (nx + 1) * ny : nx * (ny + 1);
    const int f = (xface ? (int)blockIdx.x : (int)blockIdx.x - nbu) * W + c;
    const bool in = f < nf;
    double* field = (xface ? u : v) + f;

    if (r == 0) serial[c] = 0;
    __syncthreads();
    if (in) {
        int l, rr;
        if (xface) {  // remap_x_face_velocity
            const int I = f % (nx + 1), j = f / (nx + 1);
            l = (I == 0 ? 0 : I - 1) + nx * j;
            rr = I == 0 || I == nx ? l : l + 1;
        } else {  // remap_y_face_velocity
            const int i = f % nx, J = f / nx;
            l = i + nx * (J == 0 ? 0 : J - 1);
            rr = J == 0 || J == ny ? l : l + nx;
        }
        const bool edge = l == rr;
        bool ok = true;
#pragma unroll 4
        for (int k = ka; k < kb; ++k) {
            const int o = n2 * k;
            const double a = __ldg(h_old + l + o), b = __ldg(target_h + l + o);
            const double a2 = __ldg(h_old + rr + o), b2 = __ldg(target_h + rr + o);
            const double x = field[nf * k];
            ok = ok && finite(x);
            t.at(T::D, k) = edge ? a : 0.5 * (a + a2);
            t.at(DZ, k) = edge ? b : 0.5 * (b + b2);
            t.at(T::Q(0), k) = x;
        }
        if (!ok) serial[c] = 1;
    }
    __syncthreads();
    if (r < 2 && in) {  // old depths on one row of threads, new depths on the next
        const int x = r == 0 ? T::D : DZ, z = r == 0 ? T::ZO : T::ZN;
        double s = 0.0;
        bool mono = true;
        t.at(z, 0) = 0.0;
#pragma unroll 4
        for (int k = 0; k < nz; ++k) {
            const double y = t.at(x, k);
            mono = mono && y >= 0.0;
            s = s + y;
            t.at(z, k + 1) = s;
        }
        if (!mono) serial[c] = 1;
    }
    __syncthreads();
    const bool ser = in && serial[c];
    if (in && !ser) tile_positions(t, nz, W, ka, kb == nz && ka < kb ? nz + 1 : kb);
    __syncthreads();
    if (METHOD == kPPM) {
        Halo h{};
        if (in && !ser) h = tile_halo(t, 0, nz, ka, kb);
        __syncthreads();
        if (in && !ser) tile_parabolas(t, 0, h, nz, ka, kb);
        __syncthreads();
    } else if (METHOD == kPLM) {
        if (in && !ser) tile_slopes(t, 0, nz, ka, kb);
        __syncthreads();
    }
    if (in && !ser) {
        tile_integrals<METHOD, 1>(t, W, ka, kb, [](int) { return 0; }, [&](int k, const double(&sum)[1], int) {
            const double dzn = t.at(DZ, k);
            double val = dzn <= 0.0 ? 0.0 : sum[0] / dzn;
            if (METHOD != kPCM && nz == 1) val = t.at(T::Q(0), 0);
            if (KE)
                t.at(QN, k) = val;
            else
                field[nf * k] = val;
        });
    } else if (ser && r == 0) {
        double* out = &t.at(QN, 0);
        const Col<T::S> dz = t.col(DZ);
        serial_column<METHOD>(
            nz, t.col(T::D), [=](int k) { return dz[k]; }, t.col(T::Q(0)),
            [=](int k, double val) {
                if (KE)
                    out[k * T::S] = val;
                else
                    field[nf * k] = val;
            });
    }
    if (!KE) return;
    __syncthreads();
    if (r == 0 && in)
        rescale_anomaly_ke<T::S>(nz, t.col(T::D), t.col(DZ), [=](int k) { return field[nf * k]; }, &t.at(QN, 0));
    __syncthreads();
    if (in)
        for (int k = ka; k < kb; ++k) field[nf * k] = t.at(QN, k);
}

// -------------------------------------------------------------------- host --
int fail(int code, const std::string& msg) {
    g_err = msg;
    redi::set_last_error(msg);
    return code;
}

// Width of a tile whose columns take `column` bytes of shared memory: the widest
// of 32, 16 and 8 that leaves room for three blocks per SM. Wide tiles make long
// rows and few idle threads in the per-column sums; three blocks cover one
// another's loads and barriers. Measured (k_ale_columns of two tracers and
// k_ale_faces, us): nz = 30, W 32 / 16 / 8: 222 / 223 / 244 and 181 / 201 / 224 at
// 479x303; nz = 75: 10768 / 7750 / 6795 and 11270 / 6110 / 6690 at 1444x1084.
constexpr size_t kTileGoal = 75 * 1024;
int tile_width(size_t column) { return 32 * column <= kTileGoal ? 32 : 16 * column <= kTileGoal ? 16 : 8; }

// Threads of a block: about four layers each (3 and 5 measured within 4 % either
// way, 8 a third slower), whole warps, at least two rows of threads (the faces
// sum old and new depths on one row each).
int tile_threads(int nz, int W) {
    int G = (nz + 3) / 4;
    G = G < 2 ? 2 : G;
    const int step = 32 / W;
    G = (G + step - 1) / step * step;
    return G * W > kThreadsMax ? kThreadsMax : G * W;
}

// Every kernel is allowed kTileGoal, which no tile exceeds (nz <= 128), whatever
// the call needs: the attribute is the same from every thread.
template <class F>
cudaError_t allow_smem(F* kernel) {
    static_assert(8 * column_bytes(kNzMax, 9) <= kTileGoal, "the deepest columns in the narrowest tile");
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileGoal);
}

template <int METHOD, int W, int NT>
cudaError_t launch_columns(const ale_b200_step_args& a, const Dims& d, cudaStream_t st) {
    const size_t smem = W * column_bytes(a.nz, tile_arrays(METHOD, NT, 0));
    cudaError_t e = allow_smem(k_ale_columns<METHOD, W, NT>);
    if (e != cudaSuccess) return e;
    const int nb = (d.n2 + W - 1) / W;
    const int threads = tile_threads(a.nz, W);
    TracerSet cur{};
    int n = 0, first = 1;
    do {
        cur.n = 0;
        for (; n < a.ntracers && cur.n < kMaxTracers; ++n) {
            if (!a.tracers[n]) continue;
            cur.tr[cur.n] = a.tracers[n];
            cur.budget[cur.n++] = n == a.idx_temperature ? a.heat_budget : n == a.idx_salinity ? a.salt_budget : nullptr;
        }
        while (n < a.ntracers && !a.tracers[n]) ++n;
        redi::launch_begin(redi::K_ALE_COLUMNS, st);
        k_ale_columns<METHOD, W, NT><<<nb, threads, smem, st>>>(d, cur, first, n == a.ntracers, a.h_layer, a.bt_eta,
                                                                a.bt_H_ref, a.dsig, a.total_h, a.h_ref, a.h_old,
                                                                a.target_h, a.mass_budget);
        redi::launch_end(redi::K_ALE_COLUMNS, st);
        first = 0;
    } while (n < a.ntracers);
    return cudaSuccess;
}

template <int METHOD, int W, bool KE>
cudaError_t launch_faces(const ale_b200_step_args& a, const Dims& d, cudaStream_t st) {
    const size_t smem = W * column_bytes(a.nz, tile_arrays(METHOD, 1, KE ? 2 : 1));
    cudaError_t e = allow_smem(k_ale_faces<METHOD, W, KE>);
    if (e != cudaSuccess) return e;
    const int nu = (a.nx + 1) * a.ny, nv = a.nx * (a.ny + 1);
    const int nbu = (nu + W - 1) / W, nbv = (nv + W - 1) / W;
    const int threads = tile_threads(a.nz, W);
    redi::launch_begin(redi::K_ALE_FACES, st);
    k_ale_faces<METHOD, W, KE><<<nbu + nbv, threads, smem, st>>>(d, nbu, a.h_old, a.target_h, a.u, a.v);
    redi::launch_end(redi::K_ALE_FACES, st);
    return cudaSuccess;
}

template <int METHOD, int NT>
cudaError_t launch_columns_nt(const ale_b200_step_args& a, const Dims& d, cudaStream_t st) {
    const int W = tile_width(column_bytes(a.nz, tile_arrays(METHOD, NT, 0)));
    return W == 32   ? launch_columns<METHOD, 32, NT>(a, d, st)
           : W == 16 ? launch_columns<METHOD, 16, NT>(a, d, st)
                     : launch_columns<METHOD, 8, NT>(a, d, st);
}

template <int METHOD, bool KE>
cudaError_t launch_faces_ke(const ale_b200_step_args& a, const Dims& d, cudaStream_t st) {
    const int W = tile_width(column_bytes(a.nz, tile_arrays(METHOD, 1, KE ? 2 : 1)));
    return W == 32   ? launch_faces<METHOD, 32, KE>(a, d, st)
           : W == 16 ? launch_faces<METHOD, 16, KE>(a, d, st)
                     : launch_faces<METHOD, 8, KE>(a, d, st);
}

template <int METHOD>
int launch(const ale_b200_step_args& a, cudaStream_t st) {
    const Dims d{a.nx, a.ny, a.nz, a.nx * a.ny};
    int ntr = 0;
    for (int n = 0; n < a.ntracers; ++n) ntr += a.tracers[n] != nullptr;
    // tracers two at a time: they share the positions, and their arithmetic overlaps
    // (nz = 30: 223 us against 279 one at a time)
    cudaError_t e = ntr < 2 ? launch_columns_nt<METHOD, 1>(a, d, st) : launch_columns_nt<METHOD, 2>(a, d, st);
    if (e == cudaSuccess && a.u && a.v)
        e = a.conserve_ke ? launch_faces_ke<METHOD, true>(a, d, st) : launch_faces_ke<METHOD, false>(a, d, st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ALE_B200_E_CUDA, std::string("ale: launch: ") + cudaGetErrorString(e));
    return ALE_B200_OK;
}

int run(const ale_b200_step_args* a, cudaStream_t st) {
    if (!a) return fail(ALE_B200_E_ARG, "ale: NULL argument block");
    if (a->nx < 1 || a->ny < 1 || a->nz < 1) return fail(ALE_B200_E_ARG, "ale: nx, ny, nz must be >= 1");
    if (a->nz > kNzMax) return fail(ALE_B200_E_ARG, "ale: nz exceeds ALE_B200_NZ_MAX (the reference's NZ_STACK_MAX)");
    if ((long long)(a->nx + 1) * (a->ny + 1) * a->nz > (long long)INT_MAX - 1024)
        return fail(ALE_B200_E_ARG, "ale: domain too large for 32-bit offsets");
    if (a->method == 4 || a->method == 5)
        return fail(ALE_B200_E_UNSUPPORTED, "ale: REMAP_PPM_H4 and REMAP_PQM are not implemented");
    if (!a->h_layer || !a->mass_budget || !a->bt_eta || !a->bt_H_ref || !a->dsig || !a->h_old || !a->target_h)
        return fail(ALE_B200_E_ARG, "ale: a required array pointer is NULL");
    if (a->ntracers < 0 || (a->ntracers > 0 && !a->tracers)) return fail(ALE_B200_E_ARG, "ale: bad tracer table");
    for (int n = 0; n < a->ntracers; ++n) {
        if (!a->tracers[n]) continue;
        if ((n == a->idx_temperature && !a->heat_budget) || (n == a->idx_salinity && !a->salt_budget))
            return fail(ALE_B200_E_ARG, "ale: heat / salt budget NULL for the temperature / salinity slot");
    }
    int rc;
    if (a->method == kPCM)
        rc = launch<kPCM>(*a, st);
    else if (a->method == kPPM && a->nz > 2)
        rc = launch<kPPM>(*a, st);
    else
        rc = launch<kPLM>(*a, st);  // REMAP_PLM, the select-case default, and PPM of one or two layers
    if (rc == ALE_B200_OK) g_err.clear();
    return rc;
}

void report(const char* who, int rc) {
    if (rc < 0) std::fprintf(stderr, "%s: %s\n", who, g_err.c_str());
}

}  // namespace

extern "C" {

int ale_b200_remap_step(const ale_b200_step_args* args, void* stream) {
    return run(args, static_cast<cudaStream_t>(stream));
}

const char* ale_b200_last_error(void) { return g_err.c_str(); }

void ale_remap_cuda(int nx, int ny, int nz, int method, int fused, double* h_layer, double* h_old, double* target_h,
                    double* total_h, double* h_ref, double* hTr_t, double* hTr_s, double* u, double* v,
                    double* mass_b, double* heat_b, double* salt_b, double* eta, double* H_ref, double* dsig) {
    (void)fused;  // the reference's faithful and fused forms give the same results
    double* tr[2] = {hTr_t, hTr_s};
    const ale_b200_step_args a{nx,     ny,     nz,     method, 0,      2,     0,      1,      h_layer, tr,
                               u,      v,      mass_b, heat_b, salt_b, eta,   H_ref,  dsig,   total_h, h_ref,
                               h_old,  target_h};
    report("ale_remap_cuda", run(&a, nullptr));
}

void ale_remap_opt(int nx, int ny, int nz, double* h_layer, double* h_old, double* target_h, double* hTr_t,
                   double* hTr_s, double* u, double* v, double* mass_b, double* heat_b, double* salt_b, double* eta,
                   double* H_ref, double* dsig) {
    double* tr[2] = {hTr_t, hTr_s};
    const ale_b200_step_args a{nx,     ny,     nz,     kPPM,   0,      2,       0,      1,       h_layer, tr,
                               u,      v,      mass_b, heat_b, salt_b, eta,     H_ref,  dsig,    nullptr, nullptr,
                               h_old,  target_h};
    report("ale_remap_opt", run(&a, nullptr));
}

void cuda_sync(void) { cudaDeviceSynchronize(); }

}  // extern "C"
