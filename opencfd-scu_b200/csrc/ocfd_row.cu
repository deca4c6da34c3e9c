// ocfd_row.cu -- the UP7 walk of the x sweep, four cells a lane (sm_100a;
// FP64, and FP32 for the precision form).
//
// Same results as the reference's OCFD_dx1/2 chain on UP7 faces
// (src/OCFD_Schemes.cu:159-381, 865-907): every point is split once, du has
// one writer per element.  Cells next to any other face, and the first and
// last cells of a bounded line, go to the x list of deferred cells for the
// fix-up kernel, as in the other walks.
//
// Organisation.  A warp walks 32 / LPR rows of x, LPR lanes a row, 4 LPR
// cells of each row per pass.  Per pass every lane loads four consecutive
// points (16-byte loads; LAP-box rows start on 64-byte boundaries), splits
// them and stores the ten split values of each; then, field by field, it
// reads the 12 points that its four cells reach and forms the cells' flux
// differences from them directly (UP7 is linear: the difference of two faces
// is eight coefficients a side).  That is 12 shared-memory values a side and
// field for four cells, in 16-byte reads, where one cell a lane reads 28, and
// nothing is passed between lanes.  16-byte units of FP64 are kept even ones
// first, then odd ones, so that the lanes of a read touch consecutive units.
// The last eight points of a pass are the first eight of the next.
// Bound in FP64 by the FP64 pipe and the shared-memory one between them (45 and
// 44 % of peak at 160^3, a quarter of the warps an SM holds), in FP32 by issue (72 %).  At 160^3: 100 us in FP64 against 139 for the one-cell-a-lane
// ring.  With the marches, the sweeps of a 256^3 stage: 1.27 against 1.39 ms
// (FP64), 0.75 against 0.83 (FP32).
#include "ocfd_walk.cuh"

#include <cuda_runtime.h>

namespace ocfd {

cudaError_t launch_sweep3_fix(const Params &p, int dir, cudaStream_t st);
cudaError_t launch_sweep4_fix(const Params &p, int dir, cudaStream_t st);

namespace {

using namespace walk;

constexpr int RW = 4;          // warps per block
template <typename R> constexpr int row_blocks() { return sizeof(R) == 8 ? 4 : 6; }     // blocks per SM

template <typename R> struct Vec;
template <> struct Vec<double> { using T = double2; static constexpr int N = 2; };
template <> struct Vec<float> { using T = float4; static constexpr int N = 4; };

// split values of a warp's rows for one pass
template <typename R, int LPR>
struct RowTile {
    static constexpr int ROWS = 32 / LPR, C = 4 * LPR;        // rows a warp, cells a row and pass
    static constexpr int UNITS = (C + 8) / Vec<R>::N;          // 16-byte units a row: points x0-4 .. x0+C+3
    typename Vec<R>::T u[10][ROWS][UNITS];
    // place of unit c: FP64 even units first
    static __device__ __forceinline__ int at(int c) { return Vec<R>::N == 2 ? (c >> 1) + (c & 1) * (UNITS / 2) : c; }
};

// 420 times UP7's flux difference over cell i as coefficients of the points
// i-4 .. i+3 of the positive side; the negative side takes them negated
// and mirrored on i-3 .. i+4
template <typename R> __device__ __forceinline__ constexpr R up7_d(int k) {
    return k == 0 ? (R)3 : k == 1 ? (R)-28 : k == 2 ? (R)126 : k == 3 ? (R)-420 : k == 4 ? (R)105
         : k == 5 ? (R)252 : k == 6 ? (R)-42 : (R)4;
}

__device__ __forceinline__ void load4(const double *f, double (&v)[4]) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(f)), b = __ldg(reinterpret_cast<const double2 *>(f) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void load4(const float *f, float (&v)[4]) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(f));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
// units of four consecutive points
__device__ __forceinline__ void put_units(double2 *u, int c, int half, const double (&v)[4]) {
    u[c >> 1] = make_double2(v[0], v[1]);
    u[(c >> 1) + half] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void put_units(float4 *u, int c, int, const float (&v)[4]) {
    u[c] = make_float4(v[0], v[1], v[2], v[3]);
}
// the 12 points from unit c on
__device__ __forceinline__ void get_units(const double2 *u, int c, int half, double (&v)[12]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const double2 a = u[(c >> 1) + j], b = u[(c >> 1) + j + half];
        v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = b.x; v[4 * j + 3] = b.y;
    }
}
__device__ __forceinline__ void get_units(const float4 *u, int c, int, float (&v)[12]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const float4 a = u[c + j];
        v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = a.z; v[4 * j + 3] = a.w;
    }
}
__device__ __forceinline__ void store4(double *f, const double (&v)[4]) {
    reinterpret_cast<double2 *>(f)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(f)[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void store4(float *f, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(f) = make_float4(v[0], v[1], v[2], v[3]);
}

template <bool UNI, bool EPS0, typename R, int LPR>
__global__ void __launch_bounds__(32 * RW, row_blocks<R>()) k_row(const __grid_constant__ Params p, int seg_len) {
    using T = RowTile<R, LPR>;
    constexpr int N4 = 4 / Vec<R>::N, HALF = T::UNITS / 2;     // units of four points
    extern __shared__ __align__(16) unsigned char smem_row[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T &tile = reinterpret_cast<T *>(smem_row)[wid];
    const long long nrows = (long long)p.ny * p.nz;
    const long long r0 = ((long long)blockIdx.x * RW + wid) * T::ROWS;
    if (r0 >= nrows) return;                                   // the whole warp
    const int n = p.nx, rl = lane / LPR, il = lane % LPR;
    auto row_base = [&](long long row) {                       // LAP offset of the row's first cell
        const int j = (int)(row % p.ny), k = (int)(row / p.ny);
        return (long long)(k + OCFD_LAP) * p.zs + (long long)(j + OCFD_LAP) * p.ys + OCFD_LAP;
    };
    const bool rowok = r0 + rl < nrows;
    const long long row = rowok ? r0 + rl : nrows - 1;         // keep addresses in range
    const long long base = row_base(row);
    const int8_t *fl = p.flag[0] + (long long)(n + 1) * row;
    R *__restrict__ du = du_r<R>(p);
    const long long N = p.N, cb = (long long)n * row;
    const bool hybrid = p.scheme_invis == 310;
    const bool wide = n % 4 == 0;                              // 16-byte stores of four cells
    const R sc0 = UNI ? up7_scale((R)p.mc[M_AJAC], p.inv_h[0]) : (R)0.0;

    auto split = [&](long long o, R d, R u, R v, R w, R Tt, R (&fp)[5], R (&fm)[5]) {
        split_point<0, UNI, EPS0>(p, o, d, u, v, w, Tt, fp, fm);
    };
    const int xs = (int)blockIdx.y * seg_len, xe = xs + seg_len < n ? xs + seg_len : n;     // this segment's cells
    // points xs-4 .. xs+3 of each row, one a lane
    if (lane < 8 * T::ROWS) {
        const int rr = lane >> 3, t = lane & 7;
        const long long row2 = r0 + rr < nrows ? r0 + rr : nrows - 1;
        const long long o = row_base(row2) + xs + t - 4;
        R q5[5], fp[5], fm[5];
        load5(p, o, q5);
        split(o, q5[0], q5[1], q5[2], q5[3], q5[4], fp, fm);
#pragma unroll
        for (int m = 0; m < 5; m++) {
            reinterpret_cast<R *>(&tile.u[m][rr][T::at(t / Vec<R>::N)])[t % Vec<R>::N] = fp[m];
            reinterpret_cast<R *>(&tile.u[5 + m][rr][T::at(t / Vec<R>::N)])[t % Vec<R>::N] = fm[m];
        }
    }
    for (int x0 = xs; x0 < xe; x0 += T::C) {
        const int i0 = x0 + 4 * il;                            // the lane's cells i0 .. i0+3
        // flags of the faces i0-1/2 .. i0+7/2
        int hf[5];
#pragma unroll
        for (int t = 0; t < 5; t++)
            hf[t] = (hybrid && i0 + t <= n) ? flag_at(p, 0, fl, i0 + t) : 2;
        {
            const int P = i0 + 4;                              // the lane's new points P .. P+3
            R q[5][4];
            const long long o = OCFD_IDX(p, base + P, p.lapN);
            if (P <= n + 3) {
#pragma unroll
                for (int m = 0; m < 5; m++) load4(prim_r<R>(p, m) + o, q[m]);
            } else {
#pragma unroll
                for (int m = 0; m < 5; m++)
#pragma unroll
                    for (int t = 0; t < 4; t++) q[m][t] = (R)1.0;
            }
            R fp[5][4], fm[5][4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                R a[5], b[5];
                // (points past the last ghost are not used; their metrics are not read)
                split(P + t <= n + 3 ? o + t : base, q[0][t], q[1][t], q[2][t], q[3][t], q[4][t], a, b);
#pragma unroll
                for (int m = 0; m < 5; m++) { fp[m][t] = a[m]; fm[m][t] = b[m]; }
            }
#pragma unroll
            for (int m = 0; m < 5; m++) {
                put_units(tile.u[m][rl], N4 * (il + 2), HALF, fp[m]);
                put_units(tile.u[5 + m][rl], N4 * (il + 2), HALF, fm[m]);
            }
        }
        __syncwarp();
        // cells beside a face that is not UP7, and line ends, are left to the fix-up
        unsigned late = 0;
        if (rowok) {
            bool slow[5];
#pragma unroll
            for (int t = 0; t < 5; t++) slow[t] = !up7_face(p, hf[t]) || near_closure(p, 0, i0 + t - 1, n);
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (i0 + t < n && (slow[t] || slow[t + 1] || (p.has_bnd && rule_cell(p, 0, i0 + t, n)))) late |= 1u << t;
        }
        if (__any_sync(FULL, late != 0)) {
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const unsigned mask = __ballot_sync(FULL, (late >> t) & 1u);
                if (mask) {                                    // one atomic per warp
                    const int leader = __ffs(mask) - 1;
                    unsigned slot = 0;
                    if (lane == leader) slot = atomicAdd(p.defer_count, (unsigned)__popc(mask));
                    slot = __shfl_sync(FULL, slot, leader);
                    if ((late >> t) & 1u)
                        p.defer[0][OCFD_IDX(p, (long long)slot + __popc(mask & ((1u << lane) - 1u)), N)] = (unsigned)(cb + i0 + t);
                }
            }
        }
        R sc[4];
#pragma unroll
        for (int t = 0; t < 4; t++)
            sc[t] = UNI ? sc0 : up7_scale((R)metric<UNI>(p, M_AJAC, i0 + t < n ? base + i0 + t : base), p.inv_h[0]);
#pragma unroll
        for (int m = 0; m < 5; m++) {
            R a[12], b[12], d[4];
            get_units(tile.u[m][rl], N4 * il, HALF, a);
            get_units(tile.u[5 + m][rl], N4 * il, HALF, b);
#pragma unroll
            for (int t = 0; t < 4; t++) {
                R s = up7_d<R>(0) * a[t];
                s = fma_r(-up7_d<R>(7), b[t + 1], s);
#pragma unroll
                for (int k = 1; k < 8; k++) {
                    s = fma_r(up7_d<R>(k), a[t + k], s);
                    s = fma_r(-up7_d<R>(7 - k), b[t + k + 1], s);
                }
                d[t] = sc[t] * s;
            }
            R *out = du + m * N + cb + i0;
            if (rowok) {
                // (a deferred cell's value is overwritten by the fix-up)
                if (wide) {
                    if (i0 < n) store4(out, d);
                } else {
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        if (i0 + t < n) out[t] = d[t];
                }
            }
        }
        if (x0 + T::C < xe) {      // points x0+C-4 .. x0+C+3 open the next pass
            __syncwarp();
            constexpr int NU = 8 / Vec<R>::N, M = 10 * T::ROWS * NU;
#pragma unroll
            for (int e = lane; e < (M + 31) / 32 * 32; e += 32) {
                if (e < M) {
                    const int u = e % NU, r = e / NU % T::ROWS, sv = e / (NU * T::ROWS);
                    tile.u[sv][r][T::at(u)] = tile.u[sv][r][T::at(T::C / Vec<R>::N + u)];
                }
            }
            __syncwarp();
        }
    }
}

template <bool UNI, bool EPS0, typename R, int LPR>
cudaError_t set_smem() {
    return cudaFuncSetAttribute(k_row<UNI, EPS0, R, LPR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(RW * sizeof(RowTile<R, LPR>)));
}
template <bool UNI, bool EPS0, typename R>
cudaError_t prepare_r() {
    cudaError_t e = set_smem<UNI, EPS0, R, 32>();
    if (e == cudaSuccess) e = set_smem<UNI, EPS0, R, 16>();
    if (e == cudaSuccess) e = set_smem<UNI, EPS0, R, 8>();
    return e;
}

template <bool UNI, bool EPS0, typename R, int LPR>
cudaError_t launch_lpr(const Params &p, cudaStream_t st) {
    const long long warps = ((long long)p.ny * p.nz + 32 / LPR - 1) / (32 / LPR);
    // (segments of whole passes where the chip has slots left: a 500x12x12 UP7
    // step on metric fields takes 151 us where the rows' four passes took 215)
    const long long slots = 148LL * row_blocks<R>() * RW;
    const int passes = (p.nx + 4 * LPR - 1) / (4 * LPR), fit = (int)(warps < slots ? slots / warps : 1);
    const int len = fit >= passes ? 1 : (passes + fit - 1) / fit;              // passes a segment
    const dim3 grid((unsigned)((warps + RW - 1) / RW), (unsigned)((passes + len - 1) / len));
    k_row<UNI, EPS0, R, LPR><<<grid, 32 * RW, RW * sizeof(RowTile<R, LPR>), st>>>(p, len * 4 * LPR);
    return cudaGetLastError();
}

template <bool UNI, bool EPS0, typename R>
cudaError_t launch_r(const Params &p, cudaStream_t st) {
    switch (row_lanes(p.nx, (long long)p.ny * p.nz, 148LL * row_blocks<R>() * RW)) {
    case 32: return launch_lpr<UNI, EPS0, R, 32>(p, st);
    case 16: return launch_lpr<UNI, EPS0, R, 16>(p, st);
    default: return launch_lpr<UNI, EPS0, R, 8>(p, st);
    }
}

template <typename R>
cudaError_t launch_row_r(const Params &p, cudaStream_t st) {
    if (p.uniform_metrics)
        return p.epsl_sw == 0.0 ? launch_r<true, true, R>(p, st) : launch_r<true, false, R>(p, st);
    return launch_r<false, false, R>(p, st);
}

}  // namespace

// the shared-memory size of every instance, set on the current device
// before the first launch (and before any stream capture)
cudaError_t row_prepare() {
    cudaError_t e = cudaSuccess;
    auto one = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    one(prepare_r<true, true, double>()); one(prepare_r<true, false, double>()); one(prepare_r<false, false, double>());
    one(prepare_r<true, true, float>());  one(prepare_r<true, false, float>());  one(prepare_r<false, false, float>());
    return e;
}

// the x sweep of the UP7 walk, then the fix-up of its deferred cells (the
// caller clears the deferred counters)
cudaError_t launch_row(const Params &p, cudaStream_t st) {
    const cudaError_t e = p.mixed ? launch_row_r<float>(p, st) : launch_row_r<double>(p, st);
    if (e != cudaSuccess) return e;
    return p.mixed ? launch_sweep4_fix(p, 0, st) : launch_sweep3_fix(p, 0, st);
}

}  // namespace ocfd
