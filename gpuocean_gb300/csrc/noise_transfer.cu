// Stand-alone transfer of the SOAR coarse field to the ocean state (single
// simulator, and batched for moments outside the fused ensemble step):
// bicubic up-sampling + geostrophic balance, K/ocean_noise.cu:256-666.
//
// Compiled with the ensemble step's arithmetic options (no FMA contraction),
// so that these kernels and the fused step epilogue, which both use
// noise_transfer.cuh, round identically.
#include "noise_transfer.cuh"

namespace goc {

constexpr int kPR = kPY / kPT;   // cells per thread
// shared scratch of one tile: the coefficient matrices of up to 12 x 12
// coarse cells (factors >= 4 for the 34 fine cells of a tile + ring) and the
// per-column / per-row coarse indices and fractions
constexpr int kScratch = 12 * 12 * 17 + 2 * ((kPX + 2) + (kPY + 2));

// One kPX x kPY tile of interior cells (tile origin bx, by in interior
// cells).  Each thread owns kPR cells of one column; their state is loaded
// first so that the loads overlap the perturbation field (the corner depths,
// shared by the members and L2-resident, are read when used).
__device__ void perturb_tile(const GocNoiseDesc& d, const OceanRef& o, int bx, int by) {
    __shared__ float s_de[kPY + 2][kPX + 2];
    __shared__ float s_scratch[kScratch];
    const int tx = threadIdx.x, t = threadIdx.y * kPX + tx;
    constexpr int NT = kPX * kPT;
    const bool factor1 = d.interpolation_factor <= 1;
    const int ti = 2 + bx + tx;
    float q[kPR][3];
#pragma unroll
    for (int r = 0; r < kPR; ++r) {
        const int tj = 2 + by + threadIdx.y + r * kPT;
        q[r][0] = q[r][1] = q[r][2] = 0.0f;
        if (ti < o.nx + 2 && tj < o.ny + 2) {
            const size_t k = (size_t)tj * o.pitch + ti;
            q[r][0] = o.eta[k];
            q[r][1] = o.hu[k];
            q[r][2] = o.hv[k];
        }
    }
    // d_eta on the tile + 1 ring (interior origin at ghost offset 2)
    noise_tile_field<kPX + 2, kPY + 2, NT>(d, o.dx, o.dy, 2 + bx - 1, 2 + by - 1, &s_de[0][0], s_scratch, kScratch, t);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPR; ++r) {
        const int tj = 2 + by + threadIdx.y + r * kPT;
        if (ti < o.nx + 2 && tj < o.ny + 2) {
            const float* h0 = o.Hi + (size_t)tj * o.hi_pitch + ti;
            const float hc[4] = {__ldg(h0), __ldg(h0 + 1), __ldg(h0 + o.hi_pitch), __ldg(h0 + o.hi_pitch + 1)};
            float e = q[r][0], u = q[r][1], v = q[r][2];
            perturbed_state(d, o.nx, o.ny, o.dx, o.dy, o.land, ti, tj, factor1,
                            [&](int jj, int ii) { return s_de[jj - (2 + by) + 1][ii - (2 + bx) + 1]; }, e, u, v, hc);
            store_cell(o, ti, tj, e, u, v);
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kPX * kPT, 3) perturb_kernel(GocNoiseDesc d, OceanRef o) {
    perturb_tile(d, o, blockIdx.x * kPX, blockIdx.y * kPY);
}

__device__ __forceinline__ OceanRef perturbed_ocean(const GocMemberDesc& m, int set) {
    return OceanRef{m.p.nx, m.p.ny, m.p.dx, m.p.dy, m.eta[set], m.hu[set], m.hv[set], m.pitch / 4, m.Hi,
                    m.Hi_pitch / 4, m.p.land_value, m.p.bc_north == 2, m.p.bc_east == 2};
}

__global__ void __launch_bounds__(kPX * kPT, 3)
perturb_batched_kernel(const GocNoiseDesc* __restrict__ nd, const GocMemberDesc* __restrict__ mem,
                       const int4* __restrict__ items, const int* __restrict__ nsub, int substep) {
    const int4 it = items[blockIdx.x];
    int set;
    if (!member_set(nsub, it.x, substep, &set)) return;
    perturb_tile(nd[it.x], perturbed_ocean(mem[it.x], set), it.y * kPX, it.z * kPY);
}

// ---- factors >= 5 on a Coriolis plane: warps that march ----

// A warp owns kPW columns (and one more on each side, whose perturbation its
// neighbours read by shuffle) and marches kPRows rows north, so that the
// perturbation of a cell is evaluated once, in registers.
constexpr int kPW = 30, kPNT = 256;
constexpr int kPWX = kRX / kPW, kPWY = kPNT / 32 / kPWX;     // warps of a tile
constexpr int kFX = kRX + 2;                                // fine columns of a tile and its ring
constexpr int kPRows = kRY / kPWY, kFY = kRY + 2;           // rows of a warp, fine rows
// coarse columns and rows under a tile and its ring that the tables have room
// for (perturb_by_rows)
constexpr int kPC = kRowsCoarseX, kPCY = kRowsCoarseY;

struct PerturbTables {
    float4 A[kPC * kPCY][5];                           // columns of the coefficient matrices (odd stride: no bank conflicts)
    float4 row[kFY][kPC];                        // A yv: the polynomial in rx of a coarse column on a fine row
    int ci[kFX], cj[kFY];
    float rx[kFX], ry[kFY];
};

// The polynomials in rx on every fine row of the tile, with the roundings of
// bicubic_eval.  A fine row crosses a coarse cell in several fine cells
// (`interpolation_factor` of them), for which the sum over powers of ry is
// the same: it is taken once per row and coarse column.
__device__ __forceinline__ void perturb_rows(const GocNoiseDesc& d, float dx, float dy, int gi0, int gj0,
                                             PerturbTables& tab, int t) {
    if (t < kFX) tab.ci[t] = bicubic_ci(d, dx, gi0 + t, &tab.rx[t]);
    for (int j = kPNT - 1 - t; j < kFY; j += kPNT) tab.cj[j] = bicubic_cj(d, dy, gj0 + j, &tab.ry[j]);
    __syncthreads();
    const int ci0 = tab.ci[0], ncx = min(tab.ci[kFX - 1] - ci0 + 1, kPC);
    const int cj0 = tab.cj[0], ncy = min(tab.cj[kFY - 1] - cj0 + 1, kPCY);
    // four threads a cell, one column of its matrix each
    for (int c = t / 4; c < ncx * ncy; c += kPNT / 4)
        tab.A[c][t % 4] = bicubic_column(d, ci0 + c % ncx, cj0 + c / ncx, t % 4);
    __syncthreads();
    for (int e = t; e < kFY * ncx; e += kPNT) {
        const int j = e / ncx, cx = e - j * ncx, cy = clampi(tab.cj[j] - cj0, 0, ncy - 1);
        float4 A[4];                            // columns
#pragma unroll
        for (int k = 0; k < 4; ++k) A[k] = tab.A[cy * ncx + cx][k];
        const float y = tab.ry[j], y2 = y * y, y3 = y * y * y;
        tab.row[j][cx] = make_float4(A[0].x * 1.0f + A[1].x * y + A[2].x * y2 + A[3].x * y3,
                                     A[0].y * 1.0f + A[1].y * y + A[2].y * y2 + A[3].y * y3,
                                     A[0].z * 1.0f + A[1].z * y + A[2].z * y2 + A[3].z * y3,
                                     A[0].w * 1.0f + A[1].w * y + A[2].w * y2 + A[3].w * y3);
    }
    __syncthreads();
}

// A lane's place in a tile with origin bx, by (interior cells).
struct PerturbLane {
    int bx, by, lane, wx, wy, i, j0, ti, tj0;   // i, j0: fine column, first fine row (of the ring)
    bool mine;                                  // owns a column of interior cells
    __device__ __forceinline__ PerturbLane(const OceanRef& o, int bx_, int by_)
        : bx(bx_), by(by_), lane(threadIdx.x), wx(threadIdx.y % kPWX), wy(threadIdx.y / kPWX), i(wx * kPW + lane),
          j0(wy * kPRows), ti(2 + bx - 1 + i), tj0(2 + by + j0), mine(lane >= 1 && lane <= kPW && ti < o.nx + 2) {}
};

// The lane's cells: state and corner depths (west corners).
struct PerturbCells {
    float q[kPRows][3], h[kPRows + 1];
    __device__ __forceinline__ PerturbCells(const OceanRef& o, const PerturbLane& L) {
#pragma unroll
        for (int r = 0; r <= kPRows; ++r) {
            h[r] = 0.0f;
            if (L.ti <= o.nx + 2 && L.tj0 + r <= o.ny + 2) h[r] = __ldg(o.Hi + ((L.tj0 + r) * o.hi_pitch + L.ti));
        }
#pragma unroll
        for (int r = 0; r < kPRows; ++r) {
            q[r][0] = q[r][1] = q[r][2] = 0.0f;
            if (L.mine && L.tj0 + r < o.ny + 2) {
                const int k = (L.tj0 + r) * o.pitch + L.ti;
                q[r][0] = o.eta[k];
                q[r][1] = o.hu[k];
                q[r][2] = o.hv[k];
            }
        }
    }
};

// Perturbs and stores the cells of a lane.
__device__ __forceinline__ void perturb_march(const GocNoiseDesc& d, const OceanRef& o, const PerturbTables& tab,
                                              const PerturbLane& L, PerturbCells& cells) {
    const int ti = L.ti;
    auto& q = cells.q;
    auto& h = cells.h;
    const int cx = clampi(tab.ci[L.i] - tab.ci[0], 0, min(tab.ci[kFX - 1] - tab.ci[0], kPC - 1));
    const float rx = tab.rx[L.i];
    const float rx2 = rx * rx, rx3 = rx * rx * rx;
    // the perturbation of eta in the lane's column, fine row j of the tile
    auto eta_at = [&](int j) {
        const float4 g = tab.row[j][cx];
        float v = 0.0f;
        v += 1.0f * g.x;
        v += rx * g.y;
        v += rx2 * g.z;
        v += rx3 * g.w;
        return v;
    };
    // reciprocals of the steps: at most 1.5 ulp a quotient, the division's 2
    const float x2 = 1.0f / (2.0f * o.dx), y2 = 1.0f / (2.0f * o.dy), land = o.land;
    const float fx = (ti + 0.5f) * o.dx * d.north_x;
    float south = eta_at(L.j0), here = eta_at(L.j0 + 1);
    float hE = __shfl_down_sync(~0u, h[0], 1), hsum = h[0] + hE;
    bool dry = h[0] == land || hE == land;
#pragma unroll
    for (int r = 0; r < kPRows; ++r) {
        const int tj = L.tj0 + r;
        const float north = eta_at(L.j0 + r + 2);
        const float west = __shfl_up_sync(~0u, here, 1), east = __shfl_down_sync(~0u, here, 1);
        hE = __shfl_down_sync(~0u, h[r + 1], 1);
        const bool dry_n = h[r + 1] == land || hE == land;
        const float H_mid = 0.25f * (hsum + h[r + 1] + hE);
        const float cor = d.f + d.beta * (fx + (tj + 0.5f) * o.dy * d.north_y);
        const float gc = __fdividef(d.g, cor);
        const float gH = gc * (H_mid + here);
        if (!(dry || dry_n)) {
            q[r][0] += here;
            q[r][1] -= gH * ((north - south) * y2);
            q[r][2] += gH * ((east - west) * x2);
        }
        if (L.mine && tj < o.ny + 2) {
            const int k = tj * o.pitch + ti;
            o.eta[k] = q[r][0];
            o.hu[k] = q[r][1];
            o.hv[k] = q[r][2];
        }
        south = here;
        here = north;
        hsum = h[r + 1] + hE;
        dry = dry_n;
    }
    // periodic ghost images
    const bool near_x = o.images_ew && (L.bx + L.wx * kPW < 4 || L.bx + (L.wx + 1) * kPW + 2 >= o.nx);
    const bool near_y = o.images_ns && (L.tj0 < 4 || L.tj0 + kPRows > o.ny);
    if ((near_x || near_y) && L.mine) {
#pragma unroll
        for (int r = 0; r < kPRows; ++r)
            if (L.tj0 + r < o.ny + 2) store_images(o, ti, L.tj0 + r, q[r][0], q[r][1], q[r][2]);
    }
}

// One tile of kRX x kRY interior cells (origin bx, by in interior cells).
//
// What bounds it: instruction issue and the latency of a tile's chain of
// loads and tables (HBM would allow twice the rate).  96 members of 512 x
// 300, factor 8: 120 us; perturb_tile, whose cells each evaluate
// the full polynomial and pass it on in shared memory, takes 193 us.  8 rows
// a warp with 80 registers (3 blocks an SM): with 4 rows and 64 registers it
// is 126 us, and more blocks spill.
__device__ __forceinline__ void perturb_rows_tile(const GocNoiseDesc& d, const OceanRef& o, int bx, int by) {
    __shared__ PerturbTables tab;
    const PerturbLane L(o, bx, by);
    PerturbCells cells(o, L);   // first: the loads overlap the tables
    perturb_rows(d, o.dx, o.dy, 2 + bx - 1, 2 + by - 1, tab, threadIdx.y * 32 + L.lane);
    if (bx + L.wx * kPW < o.nx) perturb_march(d, o, tab, L, cells);
}

__global__ void __launch_bounds__(kPNT, 3) perturb_rows_kernel(GocNoiseDesc d, OceanRef o) {
    perturb_rows_tile(d, o, blockIdx.x * kRX, blockIdx.y * kRY);
}

__global__ void __launch_bounds__(kPNT, 3)
perturb_rows_batched_kernel(const GocNoiseDesc* __restrict__ nd, const GocMemberDesc* __restrict__ mem,
                            const int4* __restrict__ items, const int* __restrict__ nsub, int substep) {
    const int4 it = items[blockIdx.x];
    int set;
    if (!member_set(nsub, it.x, substep, &set)) return;
    const GocNoiseDesc d = nd[it.x];   // its loads in one go
    perturb_rows_tile(d, perturbed_ocean(mem[it.x], set), it.y * kRX, it.z * kRY);
}

int launch_perturb_batched(const GocNoiseDesc* noise, const GocMemberDesc* members, const int4* items, int n_items,
                           int n_rows, const int* nsub, int substep, cudaStream_t stream) {
    if (n_items > 0) {
        perturb_batched_kernel<<<n_items, dim3(kPX, kPT), 0, stream>>>(noise, members, items, nsub, substep);
        count_launch();
    }
    if (n_rows > 0) {
        perturb_rows_batched_kernel<<<n_rows, dim3(32, kPNT / 32), 0, stream>>>(noise, members, items + n_items, nsub,
                                                                                substep);
        count_launch();
    }
    return check_launch("perturb_batched_kernel");
}

}  // namespace goc

using namespace goc;

static int check_transfer(const GocNoiseDesc* d) {
    if (!d) return set_error(GOC_ERR_ARG, "goc_perturb_ocean: null noise descriptor");
    if (d->coarse_nx < 1 || d->coarse_ny < 1 || !(d->coarse_dx > 0) || !(d->coarse_dy > 0) || !d->coarse ||
        d->coarse_pitch < (d->coarse_nx + 4) * 4 || d->interpolation_factor < 1)
        return set_error(GOC_ERR_ARG, "goc_perturb_ocean: bad coarse grid");
    return GOC_OK;
}

extern "C" int goc_perturb_ocean(const GocNoiseDesc* d, int nx, int ny, float dx, float dy, float* eta, float* hu,
                                 float* hv, int pitch, const float* Hi, int Hi_pitch, float land_value,
                                 int periodic_ghosts, void* stream) {
    int rc = check_transfer(d);
    if (rc) return rc;
    OceanRef o;
    if ((rc = make_ocean(nx, ny, dx, dy, eta, hu, hv, pitch, Hi, Hi_pitch, land_value,
                         periodic_ghosts && d->periodic_ns, periodic_ghosts && d->periodic_ew, &o, "goc_perturb_ocean")))
        return rc;
    if (perturb_by_rows(*d, dx, dy, ny, pitch, Hi_pitch)) {
        dim3 blk(32, kPNT / 32), grd((nx + kRX - 1) / kRX, (ny + kRY - 1) / kRY);
        perturb_rows_kernel<<<grd, blk, 0, as_stream(stream)>>>(*d, o);
        count_launch();
        return check_launch("perturb_rows_kernel");
    }
    dim3 blk(kPX, kPT), grd((nx + kPX - 1) / kPX, (ny + kPY - 1) / kPY);
    perturb_kernel<<<grd, blk, 0, as_stream(stream)>>>(*d, o);
    count_launch();
    return check_launch("perturb_kernel");
}
