// ocfd_march.cu -- the UP7 walk of the y and z sweeps as per-lane marches
// (sm_100a; FP64, and FP32 for the precision form).
//
// Same results as the UP7 walk of ocfd_sweep3.cu (the reference's
// OCFD_d{y,z}1/2 chain with the hybrid scheme's UP7 faces, src/OCFD_Schemes.cu:159-381,
// 865-907): every point split once, every face's flux formed once, one
// writer per du element.
//
// Organisation.  A warp owns 32 consecutive x columns of one z (y sweep) or
// y (z sweep) and a segment of the line; each lane walks its own column.  UP7
// is linear, so the lane keeps no window of split values: it keeps the
// running sums of the eight faces that the newest point still reaches
// (5 fields each, both signs in one sum), adds the point's split values to
// all of them and takes the finished one.  The 8-point body is unrolled, so a
// face's slot is a compile-time index.  That is 40 values of state where the
// window took 75, and 15 multiply-adds a field and cell where the two
// quotients of each face took 34 operations.
// Primitives, the cell's du and (curvilinear grids) the metrics are copied
// to the lane's own shared-memory slots by cp.async STAGES - 1 points ahead; a
// lane reads only what it copied, so the walk takes no barrier at all.
// Bounds at 160^3: FP64 by memory latency and bandwidth (120 B a cell and direction,
// 51 to 55 % of DRAM peak with 12 warps an SM), FP32 by instruction issue (70 %).
// At 160^3, y / z: FP64 110 / 108 us against 158 / 171 for the ring walk; FP32
// 78 / 79 us against 112 / 107 for a march over tiles from the tensor copy
// engine with a register window of split values.
//
// Faces that are not plain UP7 (hybrid flags other than 1, faces within
// reach of a boundary closure) defer the cells on both sides, and the first
// and last cells of a bounded line, to the same per-direction lists the
// ring walk uses; the fix-up kernel recomputes them.
#include "ocfd_tma.cuh"
#include "ocfd_walk.cuh"

#include <cuda_runtime.h>

namespace ocfd {

cudaError_t launch_sweep3_fix(const Params &p, int dir, cudaStream_t st);
cudaError_t launch_sweep4_fix(const Params &p, int dir, cudaStream_t st);

namespace {

using namespace walk;

constexpr int MW = 4;          // warps per block
constexpr int STAGES = 4;      // points in flight or in use per lane

__device__ __forceinline__ void copy_async(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(tma::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(tma::smem_u32(dst)), "l"(src) : "memory");
}

// values staged per point: 5 primitives and 5 du, and on a curvilinear grid
// the point's metric row and the cell's Jacobian (FP64 in both forms)
template <bool UNI, typename R>
struct Stage {
    R q[10][32 * MW];
    double met[UNI ? 1 : 4][UNI ? 1 : 32 * MW];
};

// blocks per SM the register budget is fitted to
template <typename R> constexpr int march_blocks() { return sizeof(R) == 8 ? 3 : 5; }

template <int DIR, bool UNI, bool EPS0, typename R>
__global__ void __launch_bounds__(32 * MW, march_blocks<R>()) k_march(const __grid_constant__ Params p, int seg_len) {
    static_assert(DIR == 1 || DIR == 2, "the march covers the y and z sweeps");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Stage<UNI, R> *stage = reinterpret_cast<Stage<UNI, R> *>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31;
    const int ngx = (p.nx + 31) / 32;
    const int n3 = DIR == 1 ? p.nz : p.ny;
    const long long grp = (long long)blockIdx.x * MW + (tid >> 5);
    if (grp >= (long long)ngx * n3) return;                   // the whole warp
    const int g = (int)(grp % ngx), c3 = (int)(grp / ngx);
    const int x = g * 32 + lane;
    const bool colok = x < p.nx;
    const int xs = colok ? x : p.nx - 1;                      // keep addresses in range
    const int n = DIR == 1 ? p.ny : p.nz;
    const int y0 = blockIdx.y * seg_len;
    const int y1 = min(n, y0 + seg_len);
    long long base, sd, cb, cst, fst;
    const int8_t *fl;
    if (DIR == 1) {
        base = (long long)(xs + OCFD_LAP) + (long long)OCFD_LAP * p.ys + (long long)(c3 + OCFD_LAP) * p.zs;
        sd = p.ys;
        cb = (long long)xs + (long long)p.nx * p.ny * c3; cst = p.nx;
        fl = p.flag[1] + (long long)xs + (long long)p.nx * (p.ny + 1) * c3; fst = p.nx;
    } else {
        base = (long long)(xs + OCFD_LAP) + (long long)(c3 + OCFD_LAP) * p.ys + (long long)OCFD_LAP * p.zs;
        sd = p.zs;
        cb = (long long)xs + (long long)p.nx * c3; cst = (long long)p.nx * p.ny;
        fl = p.flag[2] + (long long)xs + (long long)p.nx * c3; fst = (long long)p.nx * p.ny;
    }
    R *__restrict__ du = du_r<R>(p);
    const long long N = p.N;
    const bool hybrid = p.scheme_invis == 310;
    const R sc0 = UNI ? up7_scale((R)p.mc[M_AJAC], p.inv_h[DIR]) : (R)0.0;

    // points P0 .. y1+3; point P is staged in slot (P - P0) % STAGES.  The
    // offsets run along with the walk (formed from P, the unrolled body's
    // eight of each would all stay in registers).
    const int P0 = y0 - 4, P1 = y1 + 3;
    long long of = base + (long long)P0 * sd;                 // LAP offset of the next point to fetch
    long long cf = cb + (long long)(y0 - 4 - 4) * cst;        // and the cell it completes
    long long cs = cf;                                        // the cell that the current point completes
    const int8_t *fp_ = fl + (long long)(y0 - 7) * fst;       // flag of the face that the next point completes
    auto fetch = [&](int P, int s) {
        if (P <= P1) {
            Stage<UNI, R> &S = stage[s];
            const long long o = OCFD_IDX(p, of, p.lapN);
#pragma unroll
            for (int m = 0; m < 5; m++) copy_async(&S.q[m][tid], prim_r<R>(p, m) + o);
            if constexpr (!UNI) {
#pragma unroll
                for (int m = 0; m < 3; m++) copy_async(&S.met[m][tid], p.met[M_AKX + 3 * DIR + m] + o);
            }
            if (P - 4 >= y0) {
                const long long ci = OCFD_IDX(p, cf, N);
#pragma unroll
                for (int m = 0; m < 5; m++) copy_async(&S.q[5 + m][tid], du + m * N + ci);
                if constexpr (!UNI) copy_async(&S.met[3][tid], p.met[M_AJAC] + OCFD_IDX(p, of - 4 * sd, p.lapN));
            }
        }
        of += sd;
        cf += cst;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // flag of face F+1/2, F = P - 4, is entry F+1 = P - 3
    auto next_flag = [&](int P) {
        const int e = P - 3;
        const int8_t *f = fp_;
        fp_ += fst;
        return (hybrid && e >= y0 && e <= y1) ? flag_at(p, DIR, f, 0) : 2;
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) fetch(P0 + s, s);
    int hf[4];                           // flags of points P .. P+2, loaded three points ahead
#pragma unroll
    for (int s = 0; s < 3; s++) hf[s] = next_flag(P0 + s);
    hf[3] = 2;

    R S[8][5];                           // face F's sum in slot (F - P0 + 4) % 8
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int m = 0; m < 5; m++) S[j][m] = (R)0.0;
    int prv_slow = 0;

    for (int Pc = P0; Pc <= P1; Pc += 8) {
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int P = Pc + t;
            if (P <= P1) {
                fetch(P + STAGES - 1, (t + STAGES - 1) % STAGES);
                hf[(t + 3) & 3] = next_flag(P + 3);
                asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
                const Stage<UNI, R> &G = stage[t % STAGES];
                R q[5], fp[5], fm[5];
#pragma unroll
                for (int m = 0; m < 5; m++) q[m] = G.q[m][tid];
                if constexpr (UNI) {
                    split_point<DIR, UNI, EPS0>(p, 0, q[0], q[1], q[2], q[3], q[4], fp, fm);
                } else {
                    const R cc = div_const(sqrt_r(q[4]), (R)p.Ama, (R)p.inv_Ama);
                    sw_split(q[0] * (R)p.tmp0, q[1], q[2], q[3], cc, (R)G.met[0][tid], (R)G.met[1][tid],
                             (R)G.met[2][tid], (R)p.Gamma, (R)p.epsl_sw, (R)p.split_C1, (R)p.split_C3, fp, fm);
                }
                // stencil entry k of face F = P - 4 + j is point P for k = 7 - j
                const int F = P - 4;
                R diff[5];
#pragma unroll
                for (int m = 0; m < 5; m++) {
                    S[t][m] = fma_r(up7_c<R>(0), fm[m], S[t][m]);            // face F is complete
                    diff[m] = S[t][m] - S[(t + 7) & 7][m];
                    S[(t + 7) & 7][m] = up7_c<R>(0) * fp[m];                  // face F + 7 begins
#pragma unroll
                    for (int j = 1; j < 7; j++) {
                        R &s = S[(t + j) & 7][m];
                        s = fma_r(up7_c<R>(7 - j), fp[m], s);
                        s = fma_r(up7_c<R>(j), fm[m], s);
                    }
                }
                if (F >= y0 - 1) {
                    const int slow = !up7_face(p, hf[t & 3]) || near_closure(p, DIR, F, n);
                    if (F >= y0) {               // cell F: faces F-1/2 and F+1/2
                        bool defer = colok && (slow || prv_slow);
                        if (p.has_bnd) defer = defer || (colok && rule_cell(p, DIR, F, n));
                        const long long ci = OCFD_IDX(p, cs, N);
                        const unsigned mask = __ballot_sync(FULL, defer);
                        if (mask) {              // one atomic per warp
                            const int leader = __ffs(mask) - 1;
                            unsigned slot = 0;
                            if (lane == leader) slot = atomicAdd(p.defer_count + DIR, (unsigned)__popc(mask));
                            slot = __shfl_sync(FULL, slot, leader);
                            if (defer) p.defer[DIR][OCFD_IDX(p, (long long)slot + __popc(mask & ((1u << lane) - 1u)), p.N)] = (unsigned)ci;
                        }
                        if (colok && !defer) {
                            const R sc = UNI ? sc0 : up7_scale((R)G.met[UNI ? 0 : 3][UNI ? 0 : tid], p.inv_h[DIR]);
#pragma unroll
                            for (int m = 0; m < 5; m++) du[m * N + ci] = fma_r(sc, diff[m], G.q[5 + m][tid]);
                        }
                    }
                    prv_slow = slow;
                }
                cs += cst;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

template <int DIR, bool UNI, bool EPS0, typename R>
cudaError_t set_smem() {
    return cudaFuncSetAttribute(k_march<DIR, UNI, EPS0, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(STAGES * sizeof(Stage<UNI, R>)));
}

template <int DIR, bool UNI, bool EPS0, typename R>
cudaError_t launch_one(const Params &p, cudaStream_t st) {
    const int n3 = DIR == 1 ? p.nz : p.ny;
    const int n = DIR == 1 ? p.ny : p.nz;
    const long long blocks = ((long long)((p.nx + 31) / 32) * n3 + MW - 1) / MW;
    // segments of a line: a segment walks 8 points more than its cells, so
    // the split with the fewest points on the busiest SM slot
    const long long slots = 148LL * march_blocks<R>();
    int seg_len = n;
    long long best = -1;
    for (int nseg = 1; nseg <= (n + 7) / 8; nseg++) {
        const int len = (n + nseg - 1) / nseg;
        const long long rounds = (blocks * ((n + len - 1) / len) + slots - 1) / slots;
        const long long cost = rounds * (len + 8 + 4);
        if (best < 0 || cost < best) { best = cost; seg_len = len; }
    }
    const dim3 grid((unsigned)blocks, (unsigned)((n + seg_len - 1) / seg_len));
    k_march<DIR, UNI, EPS0, R><<<grid, 32 * MW, STAGES * sizeof(Stage<UNI, R>), st>>>(p, seg_len);
    return cudaGetLastError();
}

template <bool UNI, bool EPS0, typename R>
cudaError_t launch_dir_t(const Params &p, int dir, cudaStream_t st) {
    return dir == 1 ? launch_one<1, UNI, EPS0, R>(p, st) : launch_one<2, UNI, EPS0, R>(p, st);
}

}  // namespace

// The dynamic shared-memory size of every instance, set on the current
// device before the first launch (and before any stream capture).
cudaError_t march_prepare() {
    cudaError_t e = cudaSuccess;
    auto one = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    one(set_smem<1, true, true, double>());  one(set_smem<2, true, true, double>());
    one(set_smem<1, true, false, double>()); one(set_smem<2, true, false, double>());
    one(set_smem<1, false, false, double>()); one(set_smem<2, false, false, double>());
    one(set_smem<1, true, true, float>());   one(set_smem<2, true, true, float>());
    one(set_smem<1, true, false, float>());  one(set_smem<2, true, false, float>());
    one(set_smem<1, false, false, float>()); one(set_smem<2, false, false, float>());
    return e;
}

// The march covers the UP7 walk's schemes (the hybrid scheme, UP7 without
// projection) on the y and z sweeps.
bool march_supported(const Params &p, int dir) {
    const bool fast_scheme = (p.scheme_invis == 301 && !p.charteric) || p.scheme_invis == 310;
    return (dir == 1 || dir == 2) && fast_scheme && p.defer[0] != nullptr;
}

bool march_is_faster(const Params &p) {
    return walk::march_is_faster(p.nx, p.N, p.uniform_metrics != 0, p.mixed != 0);
}

// one direction: the march, then the fix-up of its deferred cells (the
// caller clears the deferred counters once per stage, as for the ring walk)
cudaError_t launch_march_dir(const Params &p, int dir, cudaStream_t st) {
    cudaError_t e;
    if (p.mixed) {
        e = p.uniform_metrics ? (p.epsl_sw == 0.0 ? launch_dir_t<true, true, float>(p, dir, st)
                                                  : launch_dir_t<true, false, float>(p, dir, st))
                              : launch_dir_t<false, false, float>(p, dir, st);
        if (e != cudaSuccess) return e;
        return launch_sweep4_fix(p, dir, st);
    }
    e = p.uniform_metrics ? (p.epsl_sw == 0.0 ? launch_dir_t<true, true, double>(p, dir, st)
                                              : launch_dir_t<true, false, double>(p, dir, st))
                          : launch_dir_t<false, false, double>(p, dir, st);
    if (e != cudaSuccess) return e;
    return launch_sweep3_fix(p, dir, st);
}

}  // namespace ocfd
