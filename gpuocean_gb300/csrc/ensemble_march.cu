// The batched ensemble kernel that marches warp pairs up column strips
// (cdklm_march.cuh).
#include "cdklm_march.cuh"
#include "ensemble.cuh"

namespace goc {

constexpr int kMarchBlocks = 8;               // strips per SM: 128 registers a thread (cdklm_march.cuh)

// Work items: runs (member, strip, first unit, units) of kMarchRows rows, then
// the drifter chunks of step k-1 (see ensemble_rk2_kernel); each CTA takes
// item blockIdx.x first and every further one from the counter.  const_f: every
// member has one Coriolis value, and a table beside it counts for nothing.
template <bool UNI>
__global__ void __launch_bounds__(kMarchThreads, kMarchBlocks)
ensemble_march_kernel(const GocCdklmParams pu, const StepConst ku, const MarchConst mu,
                      const GocMemberDesc* __restrict__ members, bool const_f, const int4* __restrict__ runs,
                      int n_runs, const float* __restrict__ dt_table, const int* __restrict__ nsub, int max_sub, int k,
                      float* const* __restrict__ drift_pos, const int4* __restrict__ drift_chunks, int n_chunks,
                      float sensitivity, float* const* __restrict__ spare, const int* __restrict__ noise_steps,
                      int* queue) {
    __shared__ MarchSmem S;
    __shared__ int s_next;
    const int n_items = n_runs + (k >= 1 ? n_chunks : 0);
    auto next_item = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) s_next = (int)gridDim.x + atomicAdd(queue, 1);
        __syncthreads();
        return s_next;
    };
    for (int item = blockIdx.x; item < n_items; item = next_item()) {
        if (item >= n_runs) {
            const int4 c = drift_chunks[item - n_runs];
            const int ns = __ldg(nsub + c.x);
            if (k - 1 >= ns) continue;
            if (spare && k == ns && k == __ldg(noise_steps + c.x) && spare[3 * c.x]) continue;
            drift_chunk(members[c.x], drift_pos[c.x], c.y, c.z, k & 1,
                        __ldg(dt_table + (size_t)c.x * max_sub + (k - 1)), sensitivity, threadIdx.x, kMarchThreads);
            continue;
        }
        const int4 t = runs[item];
        const int m = t.x;
        if (k >= __ldg(nsub + m)) continue;  // member already at the end of its block
        const GocMemberDesc& d = members[m];
        const int in = k & 1, out = in ^ 1;
        if (threadIdx.x == 0) {
            S.m.p = d.p;
            S.m.k = make_step_const(S.m.p);
            S.m.c = make_march_const(S.m.p, S.m.k);
            S.grid = MarchGrid{d.eta[in], d.hu[in], d.hv[in], d.eta[out], d.hu[out], d.hv[out], d.Hi, d.Hm,
                               const_f ? nullptr : d.p.coriolis_cell, d.pitch / 4, d.Hi_pitch / 4, d.Hm_pitch / 4,
                               d.p.coriolis_cell_pitch / 4};
        }
        __syncthreads();
        const GocCdklmParams& ps = UNI ? pu : S.m.p;
        const StepConst& ks = UNI ? ku : S.m.k;
        const MarchConst& mc = UNI ? mu : S.m.c;
        const int row0 = 2 + t.z * kMarchRows;
        march_run(ps, d.p, ks, mc, S, __ldg(dt_table + (size_t)m * max_sub + k), t.y, row0,
                           min(row0 + t.w * kMarchRows, ps.ny + 2));
    }
}

template <bool UNI>
static int march_configure_variant(int* grid_out) {
    static int grid = 0;
    if (grid == 0) {
        auto kern = ensemble_march_kernel<UNI>;
        // shared memory for kMarchBlocks strips (1 KB each is the system's),
        // the rest of the SM's memory stays L1
        cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                               (int)((sizeof(MarchSmem) + 2048) * kMarchBlocks * 100 / (228 * 1024)) + 1);
        int blocks = 0, dev = 0, sms = 0;
        if (err == cudaSuccess)
            err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, kMarchThreads, 0);
        if (err != cudaSuccess) return set_error(GOC_ERR_CUDA, "march occupancy query: %s", cudaGetErrorString(err));
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        grid = std::max(1, sms) * std::max(1, blocks);
    }
    *grid_out = grid;
    return GOC_OK;
}

template <bool UNI>
static int march_launch_variant(Ensemble* e, int k, cudaStream_t st, const FusedNoise* fn) {
    int full = 0;
    const int rc = march_configure_variant<UNI>(&full);
    if (rc) return rc;
    const int items = e->n_march + (k >= 1 ? e->n_step_chunks : 0);
    const cudaError_t qe = cudaMemsetAsync(e->d_queue, 0, sizeof(int), st);
    if (qe != cudaSuccess) return set_error(GOC_ERR_CUDA, "ensemble work counter: %s", cudaGetErrorString(qe));
    ensemble_march_kernel<UNI><<<std::min(items, full), kMarchThreads, 0, st>>>(
        e->pu, e->ku, make_march_const(e->pu, e->ku), e->d_members, e->const_f, e->d_march, e->n_march, e->d_dt,
        e->d_nsub, e->max_substeps, k, e->d_drift_pos, e->d_step_chunks, e->n_step_chunks, e->drift_sensitivity,
        fn ? fn->spare : nullptr, e->d_nsub_noise, e->d_queue);
    count_launch();
    return check_launch("ensemble_march_kernel");
}

int ensemble_march_configure(const Ensemble* e, int* grid) {
    return e->uniform ? march_configure_variant<true>(grid) : march_configure_variant<false>(grid);
}

int ensemble_march_launch(Ensemble* e, int k, cudaStream_t st, const FusedNoise* fn) {
    return e->uniform ? march_launch_variant<true>(e, k, st, fn) : march_launch_variant<false>(e, k, st, fn);
}

}  // namespace goc
