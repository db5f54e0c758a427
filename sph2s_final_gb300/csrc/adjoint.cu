// adjoint.cu -- differentiable rollout of the single-scale step (no
// counterpart in the reference).
//
// Forward: from the creation positions and given initial velocities and
// viscosity, T steps; the state is checkpointed every K steps.
// Loss: L = mean_n (G_n - target_n)^2, G the Poly6 splat of the final
// positions on the cell centres of a node grid.
// Backward: segment by segment, latest first: the hand-written adjoint kernels run
// backwards through a tape of the segment's steps (sort permutation, sorted
// positions and velocities, densities, neighbour lists, near-boundary particles),
// holding the neighbour structure of every step constant.  The tape of the last
// segment is recorded by the forward pass, the other segments are recomputed from
// their checkpoints; in both the step's own buffers are redirected into the tape.
// Memory is one segment of tape (~440 bytes per particle per step, 384 of them the
// lists, or less where that does not fit) plus T/K checkpoints.
#include <cmath>
#include <cstring>
#include <vector>
#include "adjoint_kernels.cuh"
#include "errors.h"
#include "host_params.h"
#include "single_scale_kernels.cuh"
#include "single_scale_solver.h"

using namespace sph;
using namespace sph_ss;

namespace sph {

struct Rollout {
    int T = 0, K = 0;
    float dt = 0.0f, mu = 0.0f;
    uint32_t n = 0, ncells = 0;
    std::vector<void*> owned;
    std::vector<float4*> ck_pos, ck_vel;
    std::vector<uint32_t*> perm;
    std::vector<float4*> xh, vh;
    std::vector<float*> rho;
    std::vector<float2*> aux;
    std::vector<uint4*> nbr;  // list_cap entries each
    uint32_t list_cap = kMaxNbr;
    std::vector<uint32_t*> cnt;
    std::vector<uint2*> cells;
    std::vector<uint32_t*> nlist;   // near-boundary particles, their number and flags
    std::vector<uint32_t*> ncount;
    std::vector<uint8_t*> nflag;
    float4 *gx = nullptr, *gv = nullptr, *gx2 = nullptr, *gv2 = nullptr, *lam = nullptr;
    float4* gb = nullptr;  // the boundary force's part of gx2
    float4* gxT = nullptr;
    float* grho = nullptr;
    float* gmu_part = nullptr;  // [K][blocks]
    double* gmu_acc = nullptr;
    bool forward_done = false, have_loss = false;
    // The segment whose steps the tape holds (-1: none), and the constants they
    // were computed with.  The forward pass records its last segment, which is the
    // first that the backward pass needs.
    int taped = -1;
    SimParams taped_P;
    float4 *end_pos = nullptr, *end_vel = nullptr;  // state after a rollout of one segment
};

}  // namespace sph

namespace {

template <class T>
int ralloc(Rollout* r, T** p, size_t count) {
    SPH_CUDA(cudaMalloc((void**)p, sizeof(T) * (count ? count : 1)));
    r->owned.push_back(*p);
    return SPH_OK;
}

void free_rollout(Rollout* r) {
    if (!r) return;
    for (void* p : r->owned) cudaFree(p);
    delete r;
}

int alloc_rollout(sph_solver* s, int T, int K, uint32_t list_cap, Rollout** out) {
    Rollout* r = new Rollout();
    r->list_cap = list_cap;
    r->T = T;
    r->K = K;
    r->n = s->n;
    r->ncells = s->ncells;
    const int nseg = (T + K - 1) / K;
    const uint32_t n = s->n;
    int rc = SPH_OK;
    r->ck_pos.resize(nseg);
    r->ck_vel.resize(nseg);
    for (int c = 0; c < nseg && rc == SPH_OK; ++c) {
        rc = ralloc(r, &r->ck_pos[c], n);
        if (rc == SPH_OK) rc = ralloc(r, &r->ck_vel[c], n);
    }
    r->perm.resize(K);
    r->xh.resize(K);
    r->vh.resize(K);
    r->rho.resize(K);
    r->aux.resize(K);
    r->nbr.resize(K);
    r->cnt.resize(K);
    r->cells.resize(K);
    r->nlist.resize(K);
    r->ncount.resize(K);
    r->nflag.resize(K);
    for (int k = 0; k < K && rc == SPH_OK; ++k) {
        if ((rc = ralloc(r, &r->perm[k], n)) || (rc = ralloc(r, &r->xh[k], n)) ||
            (rc = ralloc(r, &r->vh[k], n)) || (rc = ralloc(r, &r->rho[k], n)) ||
            (rc = ralloc(r, &r->aux[k], n)) || (rc = ralloc(r, &r->nbr[k], (size_t)n * (list_cap / 4))) ||
            (rc = ralloc(r, &r->cnt[k], n)) || (rc = ralloc(r, &r->cells[k], s->ncells)) ||
            (rc = ralloc(r, &r->nlist[k], n)) || (rc = ralloc(r, &r->ncount[k], 1)) ||
            (rc = ralloc(r, &r->nflag[k], n)))
            break;
    }
    const uint32_t blocks = blocks_for(n);
    if (rc == SPH_OK &&
        ((rc = ralloc(r, &r->gx, n)) || (rc = ralloc(r, &r->gv, n)) || (rc = ralloc(r, &r->gx2, n)) ||
         (rc = ralloc(r, &r->gv2, n)) || (rc = ralloc(r, &r->lam, n)) || (rc = ralloc(r, &r->gxT, n)) ||
         (rc = ralloc(r, &r->gb, n)) ||
         (rc = ralloc(r, &r->grho, n)) || (rc = ralloc(r, &r->gmu_part, (size_t)blocks * K)) ||
         (rc = ralloc(r, &r->gmu_acc, 1)) ||
         (nseg == 1 && ((rc = ralloc(r, &r->end_pos, n)) || (rc = ralloc(r, &r->end_vel, n)))))) {
    }
    if (rc != SPH_OK) {
        std::string m = sph_last_error();
        free_rollout(r);
        return fail(rc, m);
    }
    *out = r;
    return SPH_OK;
}

// One segment from the solver's state, every step recorded into the tape: the
// step's own buffers are redirected into it meanwhile.
int record_segment(sph_solver* s, int len) {
    Rollout* r = s->rollout;
    float4 *spos0 = s->spos, *svel0 = s->svel;
    float* rho0 = s->rho;
    float2* aux0 = s->aux;
    uint4* nbr0 = s->nbr;
    uint32_t* cnt0 = s->nbr_count;
    const uint32_t cap0 = s->list_cap;
    s->list_cap = r->list_cap;
    uint2* cells0 = s->cells;
    uint32_t* blist0 = s->blist;
    uint32_t* bcount0 = s->bcount;
    uint8_t* bflag0 = s->bflag;
    const int out = sort_output(s);
    uint32_t* vals0 = s->vals[out];
    for (int k = 0; k < len; ++k) {
        s->vals[out] = r->perm[k];
        s->spos = r->xh[k];
        s->svel = r->vh[k];
        s->cells_prev = s->cells;
        s->cells = r->cells[k];
        s->rho = r->rho[k];
        s->aux = r->aux[k];
        s->nbr = r->nbr[k];
        s->nbr_count = r->cnt[k];
        s->blist = r->nlist[k];
        s->bcount = r->ncount[k];
        s->bflag = r->nflag[k];
        enqueue_neighborhood(s);
        enqueue_density(s);
        enqueue_force(s, r->dt);
    }
    s->vals[out] = vals0;
    s->spos = spos0;
    s->svel = svel0;
    s->cells = cells0;
    s->cells_prev = nullptr;
    s->rho = rho0;
    s->aux = aux0;
    s->nbr = nbr0;
    s->nbr_count = cnt0;
    s->list_cap = cap0;
    s->blist = blist0;
    s->bcount = bcount0;
    s->bflag = bflag0;
    SPH_CUDA(cudaGetLastError());
    return SPH_OK;
}

// The forward pass's last segment, recorded, so that the backward pass need not
// run it again (65,536 particles, 20 steps in two segments: backward 3.39 ->
// 2.4 ms).  What the solver shows afterwards is what its own steps would have
// left: densities and cell table are copied out of the last step's record.
int advance_recorded(sph_solver* s, int seg, int len) {
    Rollout* r = s->rollout;
    if (!std::isfinite(r->dt)) return fail(SPH_E_INVALID, "sph_rollout_forward: bad dt");
    int rc = record_segment(s, len);
    if (rc != SPH_OK) return rc;
    SPH_CUDA(cudaMemcpyAsync(s->rho, r->rho[len - 1], 4 * (size_t)s->n, cudaMemcpyDeviceToDevice,
                             s->stream));
    SPH_CUDA(cudaMemcpyAsync(s->cells, r->cells[len - 1], sizeof(uint2) * s->ncells,
                             cudaMemcpyDeviceToDevice, s->stream));
    if (r->end_pos) {
        SPH_CUDA(cudaMemcpyAsync(r->end_pos, s->pos, 16 * (size_t)s->n, cudaMemcpyDeviceToDevice,
                                 s->stream));
        SPH_CUDA(cudaMemcpyAsync(r->end_vel, s->vel, 16 * (size_t)s->n, cudaMemcpyDeviceToDevice,
                                 s->stream));
    }
    s->step += (uint64_t)len;
    r->taped = seg;
    r->taped_P = s->P;
    return SPH_OK;
}

// Resets the solver to its creation positions with velocities v0 (creation
// order, host, NULL = zero).
int reset_state(sph_solver* s, const float* v0) {
    SPH_CUDA(cudaMemcpyAsync(s->pos, s->pos0, 16 * (size_t)s->n, cudaMemcpyDeviceToDevice, s->stream));
    std::vector<float4> hv(s->n);
    for (uint32_t i = 0; i < s->n; ++i)
        hv[i] = v0 ? make_float4(v0[3 * i], v0[3 * i + 1], v0[3 * i + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    SPH_CUDA(cudaMemcpyAsync(s->vel, hv.data(), 16 * (size_t)s->n, cudaMemcpyHostToDevice, s->stream));
    SPH_CUDA(cudaStreamSynchronize(s->stream));
    return SPH_OK;
}

int set_viscosity(sph_solver* s, float mu) {
    if (s->cfg.viscosity == mu) return SPH_OK;
    sph_config c = s->cfg;
    c.viscosity = mu;
    SimParams P;
    int rc = make_sim_params(c, &P);
    if (rc != SPH_OK) return rc;
    s->cfg = c;
    s->P = P;
    if (s->graph) {
        cudaGraphExecDestroy(s->graph);
        s->graph = nullptr;
    }
    return SPH_OK;
}

}  // namespace

void sph_rollout_release(sph_solver* s) {
    if (s && s->rollout) {
        free_rollout(s->rollout);
        s->rollout = nullptr;
    }
}

extern "C" {

int sph_rollout_forward(sph_solver* s, const float* v0_xyz, float viscosity, float dt,
                        int32_t steps, int32_t checkpoint_every) {
    if (!s) return fail(SPH_E_INVALID, "sph_rollout_forward: NULL handle");
    if (steps < 1 || checkpoint_every < 1 || !(dt > 0.0f) || !(viscosity >= 0.0f))
        return fail(SPH_E_INVALID, "sph_rollout_forward: need steps >= 1, checkpoint_every >= 1, dt > 0");
    if (s->n == 0) return fail(SPH_E_INVALID, "sph_rollout_forward: no fluid particles");
    const int K = checkpoint_every > steps ? steps : checkpoint_every;
    if (s->rollout && (s->rollout->T != steps || s->rollout->K != K)) sph_rollout_release(s);
    if (!s->rollout) {
        const int rc = with_list_capacity((uint64_t)s->n * K, s->list_cap, [&](uint32_t list_cap) {
            return alloc_rollout(s, steps, K, list_cap, &s->rollout);
        });
        if (rc != SPH_OK) return rc;
    }
    Rollout* r = s->rollout;
    r->dt = dt;
    r->mu = viscosity;
    r->forward_done = r->have_loss = false;
    r->taped = -1;
    int rc = set_viscosity(s, viscosity);
    if (rc != SPH_OK) return rc;
    rc = reset_state(s, v0_xyz);
    if (rc != SPH_OK) return rc;
    const int nseg = (steps + K - 1) / K;
    for (int c = 0; c < nseg; ++c) {
        SPH_CUDA(cudaMemcpyAsync(r->ck_pos[c], s->pos, 16 * (size_t)s->n, cudaMemcpyDeviceToDevice, s->stream));
        SPH_CUDA(cudaMemcpyAsync(r->ck_vel[c], s->vel, 16 * (size_t)s->n, cudaMemcpyDeviceToDevice, s->stream));
        const int len = std::min(K, steps - c * K);
        // recorded only where the backward pass's steps are the solver's own
        rc = c == nseg - 1 && s->integrator == SPH_INTEGRATOR_SYMPLECTIC_EULER && !s->force_timeout
                 ? advance_recorded(s, c, len)
                 : sph_advance(s, dt, len);
        if (rc != SPH_OK) return rc;
    }
    rc = sph_sync(s);
    if (rc != SPH_OK) return rc;
    r->forward_done = true;
    return SPH_OK;
}

int sph_rollout_density_loss(sph_solver* s, const sph_grid* nodes, const float* target,
                             float* field, double* loss) {
    if (!s || !nodes) return fail(SPH_E_INVALID, "sph_rollout_density_loss: NULL argument");
    int rc = validate_grid(*nodes, "sph_rollout_density_loss");
    if (rc != SPH_OK) return rc;
    const uint32_t nn = sph_grid_num_cells(nodes);
    const GridParams ng = make_grid_params(*nodes);
    float* d_field = nullptr;
    float* d_err = nullptr;
    float4* d_gs = nullptr;
    SPH_CUDA(cudaMalloc(&d_field, 4 * (size_t)nn));
    SPH_CUDA(cudaMalloc(&d_err, 4 * (size_t)nn));
    SPH_CUDA(cudaMalloc(&d_gs, 16 * (size_t)std::max(s->n, 1u)));
    cudaError_t e = cudaSuccess;
    std::vector<float> hf(nn);
    int out = 0;
    if (s->n) out = enqueue_neighborhood(s);
    splat_kernel<<<blocks_for(nn), 256, 0, s->stream>>>(s->spos, s->cells, s->n, s->P, ng, d_field);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hf.data(), d_field, 4 * (size_t)nn, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e == cudaSuccess && field) std::memcpy(field, hf.data(), 4 * (size_t)nn);
    if (e == cudaSuccess && target) {
        double L = 0.0;
        std::vector<float> err(nn);
        for (uint32_t k = 0; k < nn; ++k) {
            const double d = (double)hf[k] - (double)target[k];
            err[k] = (float)d;
            L += d * d;
        }
        L /= (double)nn;
        if (loss) *loss = L;
        e = cudaMemcpyAsync(d_err, err.data(), 4 * (size_t)nn, cudaMemcpyHostToDevice, s->stream);
        if (e == cudaSuccess && s->rollout && s->n) {
            const float scale = (float)(2.0 / (double)nn * 6.0 * (double)s->P.dens_coef);
            splat_grad_kernel<<<blocks_for(s->n), 256, 0, s->stream>>>(s->spos, s->n, s->P, ng,
                                                                       d_err, scale, d_gs);
            adj_unpermute_kernel<<<blocks_for(s->n), 256, 0, s->stream>>>(
                s->vals[out], s->n, d_gs, d_gs, s->rollout->gxT, s->rollout->gx2);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
            if (e == cudaSuccess) s->rollout->have_loss = true;
        }
    }
    cudaFree(d_field);
    cudaFree(d_err);
    cudaFree(d_gs);
    SPH_CUDA(e);
    return check_device_error(s);
}

int sph_rollout_backward(sph_solver* s, float* grad_v0, float* grad_x0, double* grad_mu) {
    if (!s || !s->rollout) return fail(SPH_E_INVALID, "sph_rollout_backward: no rollout");
    Rollout* r = s->rollout;
    if (!r->forward_done || !r->have_loss)
        return fail(SPH_E_INVALID, "sph_rollout_backward: run the forward and the loss first");
    const uint32_t n = s->n;
    cudaStream_t st = s->stream;
    const int nseg = (r->T + r->K - 1) / r->K;
    SPH_CUDA(cudaMemcpyAsync(r->gx, r->gxT, 16 * (size_t)n, cudaMemcpyDeviceToDevice, st));
    SPH_CUDA(cudaMemsetAsync(r->gv, 0, 16 * (size_t)n, st));
    SPH_CUDA(cudaMemsetAsync(r->gmu_acc, 0, 8, st));
    if (r->taped >= 0 && (s->force_timeout || std::memcmp(&r->taped_P, &s->P, sizeof(SimParams))))
        r->taped = -1;
    const uint32_t blocks = blocks_for(n);
    for (int c = nseg - 1; c >= 0; --c) {
        const int t0 = c * r->K, len = std::min(r->K, r->T - t0);
        const bool taped = c == r->taped;
        if (!taped || c == 0) {  // the call leaves the solver at the end of its first segment
            SPH_CUDA(cudaMemcpyAsync(s->pos, taped ? r->end_pos : r->ck_pos[c], 16 * (size_t)n, cudaMemcpyDeviceToDevice, st));
            SPH_CUDA(cudaMemcpyAsync(s->vel, taped ? r->end_vel : r->ck_vel[c], 16 * (size_t)n, cudaMemcpyDeviceToDevice, st));
        }
        if (!taped) {
            r->taped = -1;
            const int rc = record_segment(s, len);
            if (rc != SPH_OK) return rc;
        }
        for (int k = len - 1; k >= 0; --k) {  // reverse through the segment
            if (k == len - 1)
                adj_lambda_kernel<<<blocks, 256, 0, st>>>(r->gx, r->gv, r->aux[k], n, r->dt, r->lam);
            // the boundary force's adjoint beside that of the pair forces
            SPH_CUDA(cudaEventRecord(s->fork, st));
            SPH_CUDA(cudaStreamWaitEvent(s->side, s->fork, 0));
            adj_boundary_kernel<<<std::min(blocks_for(n, 256 / kBndLanes), 4u * (uint32_t)std::max(s->sms, 1)), 256, 0,
                                  s->side>>>(r->nlist[k], r->ncount[k], r->xh[k], r->lam, s->bpos,
                                             s->bcells, s->bstart, s->bcand, n, s->nb, s->P, r->gb);
            SPH_CUDA(cudaEventRecord(s->join, s->side));
            adj_force_kernel<<<blocks, 256, 0, st>>>(
                r->xh[k], r->vh[k], r->rho[k], r->nbr[k], r->cnt[k], r->cells[k], n, s->P, r->mu,
                r->dt, r->lam, r->gx, r->gv, r->gx2, r->gv2, r->grho,
                r->gmu_part + (size_t)k * blocks);
            SPH_CUDA(cudaStreamWaitEvent(st, s->join, 0));
            const AdjScatter scatter = {r->perm[k], r->gv2, k ? r->aux[k - 1] : nullptr, r->dt,
                                        r->gx, r->gv, r->lam};
            adj_density_kernel<<<blocks, 256, 0, st>>>(r->xh[k], r->nbr[k], r->cnt[k], r->cells[k],
                                                       n, s->P, r->grho, r->gb, r->nflag[k], r->gx2,
                                                       scatter);
        }
        adj_sum_kernel<<<1, 32, 0, st>>>(r->gmu_part, blocks, len, r->gmu_acc);
        SPH_CUDA(cudaGetLastError());
    }
    // gx, gv are now the adjoints of the creation-order initial state
    std::vector<float4> hg(n);
    double gm = 0.0;
    SPH_CUDA(cudaMemcpyAsync(&gm, r->gmu_acc, 8, cudaMemcpyDeviceToHost, st));
    if (grad_v0) {
        SPH_CUDA(cudaMemcpyAsync(hg.data(), r->gv, 16 * (size_t)n, cudaMemcpyDeviceToHost, st));
        SPH_CUDA(cudaStreamSynchronize(st));
        for (uint32_t i = 0; i < n; ++i) {
            grad_v0[3 * i] = hg[i].x;
            grad_v0[3 * i + 1] = hg[i].y;
            grad_v0[3 * i + 2] = hg[i].z;
        }
    }
    if (grad_x0) {
        SPH_CUDA(cudaMemcpyAsync(hg.data(), r->gx, 16 * (size_t)n, cudaMemcpyDeviceToHost, st));
        SPH_CUDA(cudaStreamSynchronize(st));
        for (uint32_t i = 0; i < n; ++i) {
            grad_x0[3 * i] = hg[i].x;
            grad_x0[3 * i + 1] = hg[i].y;
            grad_x0[3 * i + 2] = hg[i].z;
        }
    }
    SPH_CUDA(cudaStreamSynchronize(st));
    if (grad_mu) *grad_mu = gm;
    return check_device_error(s);
}

}  // extern "C"
