// The pressure solve (shaders/fluid.wgsl:381-578) as one persistent kernel per step.
//
// The reference dispatches solve_init, solve_start, then the encoded number of iterations of
// solve_q, solve_alpha, solve_update and solve_beta, every reduction a dispatch of its own, and
// keeps dispatching no-ops once the solver has switched itself off. Here one cooperative
// launch runs the whole solve and stops at convergence.
//
// Layout of the work:
//   - one warp per 4^3 block, each lane two cells of opposite red-black colour (solve_cell),
//     so the block-local Gauss-Seidel sweeps and the block's 64-wide sum tree need only warp
//     synchronisation, and every lane has a cell to update in every half-sweep;
//   - the reference sums the per-block partials with 256 strided running sums (lane l adds
//     blocks l, l + 256, ...) and then a 256-wide tree (fluid.wgsl:426-439). CTA c owns the
//     blocks b = c (mod 256) (with G < 256 CTAs, the residues c, c + G, ...), so it forms lane
//     c's running sum from its own blocks and publishes it; after a grid barrier every CTA reads
//     the 256 values and runs the same tree. All CTAs agree on alpha, beta and convergence bit for
//     bit, and the result equals the reference's order of summation;
//   - a lane keeps its cells' solver values (p, r, z, d, q, diagonal), and the warp the search
//     directions of the 96 cells across its block's faces, three a lane, which a lane advances
//     with the same expression as the cells' own lanes do. So the only cell values that cross
//     between warps are the residuals z next to block faces, once an iteration;
//   - the block's cells with the layer around them are a padded 6^3 array in shared memory
//     (SOLVE_PX, SOLVE_PY: the 32 cells of a colour in 32 banks), in which a neighbour that does
//     not count holds the value that leaves a sum as it is: -0 where neighbours are added, +0
//     where they are subtracted. No test per neighbour; between two barriers the phases are bound
//     by instruction issue (a warp's 1,109 instructions an iteration were a third of its time);
//   - a warp with one block keeps all this in registers for the whole solve; with more, in a
//     record per block (SolveRec), in shared memory while the CTA's blocks fit there and else in
//     D.wnb;
//   - the grid barrier is a counter that only grows during the launch (k_begin_step resets it): the
//     k-th barrier waits for k * (CTAs) arrivals. One atomic per CTA and a poll of the same word.
//     (Values that carry the number of their exchange and are polled themselves, no counter and no
//     fence, were slower at every size: 1M particles 108 us against 93, 66k 64 against 51; so were
//     they with clusters of 8 CTAs summing over their shared memory first, 99 and 53.)
//   - one launch can solve several simulations' systems (a batch): the CTAs split over them
//     (solve_split), each simulation's CTAs with their own barrier and sums.
// The barrier spins a bounded number of times; when it gives up it sets an error bit that the
// host reports as NTR_E_TIMEOUT, and the kernel returns.
#pragma once

#include "kernels_cells.cuh"

namespace ntr {

constexpr int SOLVE_W = 12;                 // warps per CTA
constexpr int SOLVE_T = SOLVE_W * 32;       // 384 threads
constexpr uint32_t BARRIER_SPINS = 1u << 24;
constexpr int SOLVE_XQ = 3;                 // quantities per exchange, at most

template <bool FP64>
struct SolveMath {
    using A = typename std::conditional<FP64, double, float>::type;
    static __device__ __forceinline__ A prod(float a, float b) { return FP64 ? (A)((double)a * (double)b) : (A)(a * b); }
    static __device__ __forceinline__ bool converged(double rr, double b_norm, float tol) {
        if (FP64) return sqrt(rr) <= (double)tol * fmax(b_norm, 1.0);
        return sqrtf((float)rr) <= tol * mx((float)b_norm, 1.0f);
    }
    static __device__ __forceinline__ double root(double x) { return FP64 ? sqrt(x) : (double)sqrtf((float)x); }
    static __device__ __forceinline__ double ratio(double a, double b) { return FP64 ? a / b : (double)((float)a / (float)b); }
};

// A lane's two cells of a block, one of each colour: of cells `lane` and (lane ^ 1) + 32 (two
// layers up in x and one step over in z: the other colour), k = 0 is the one of colour 0. In
// every half-sweep of the block's Gauss-Seidel each lane updates its cell of that colour.
// `lo`: cell 0 is the one of the block's lower half (cells 0-31).
struct SolveLane {
    uint32_t li[2];   // local cell
    uint32_t at[2];   // its place in the padded array
    bool lo;
    __device__ __forceinline__ explicit SolveLane(uint32_t lane);
};

// The 64-wide tree of block_sum (fluid.wgsl:414-422) over a warp whose lane holds the values
// v0, v1 of its cells: the first level adds cells l and l + 32 (the latter held by lane l ^ 1),
// the rest are shuffles. Valid in lane 0.
template <class A>
__device__ __forceinline__ A warp_tree64(const SolveLane& L, A v0, A v1) {
    const A a = L.lo ? v0 : v1, b = L.lo ? v1 : v0;
    A x = a + __shfl_xor_sync(0xffffffffu, b, 1);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, off);
    return x;
}
// Two such trees at once: after the first level lanes 0-15 go on with the first tree and lanes
// 16-31 with the second (at level 16 either order of the two terms gives the same sum). Valid in
// lane 0 (the first) and lane 16 (the second).
template <class A>
__device__ __forceinline__ A warp_tree64x2(const SolveLane& L, uint32_t lane, A u0, A u1, A v0, A v1) {
    const A x = (L.lo ? u0 : u1) + __shfl_xor_sync(0xffffffffu, L.lo ? u1 : u0, 1);
    const A y = (L.lo ? v0 : v1) + __shfl_xor_sync(0xffffffffu, L.lo ? v1 : v0, 1);
    const bool second = lane >= 16u;
    A s = (second ? y : x) + __shfl_xor_sync(0xffffffffu, second ? x : y, 16);
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
    return s;
}

// The padded array of a block: cell (x, y, z), each -1 to 4, at (x + 1) * SOLVE_PX + (y + 1) *
// SOLVE_PY + z + 1. With these strides the 32 cells of a colour, and their neighbours on one side,
// fall in 32 banks.
constexpr uint32_t SOLVE_PX = 52, SOLVE_PY = 8, SOLVE_PAD = 5 * SOLVE_PX + 5 * SOLVE_PY + 6;
__device__ __forceinline__ uint32_t solve_at(uint32_t li) { return ((li >> 4) + 1u) * SOLVE_PX + (((li >> 2) & 3u) + 1u) * SOLVE_PY + (li & 3u) + 1u; }
__device__ __forceinline__ SolveLane::SolveLane(uint32_t lane) {
    const uint32_t a = lane, b = (lane ^ 1u) + 32u;
    lo = (((a >> 4) + (a >> 2) + a) & 1u) == 0u;
    li[0] = lo ? a : b, li[1] = lo ? b : a;
    at[0] = solve_at(li[0]), at[1] = solve_at(li[1]);
}
// The cell across a face: lane's j-th of three, cell h = lane + 32 j of 96, face h / 16 (-x, +x,
// -y, +y, -z, +z). Its local cell in the neighbour block, and its place in the padded array.
__device__ __forceinline__ void solve_halo(uint32_t lane, uint32_t j, uint32_t& face, uint32_t& li, uint32_t& at) {
    const uint32_t h = lane + 32u * j, a = (h >> 2) & 3u, b = h & 3u;
    face = h >> 4;
    const uint32_t d = face >> 1, hi = face & 1u, far = hi ? 0u : 3u;
    const uint32_t x = d == 0u ? far : a, y = d == 1u ? far : d == 0u ? a : b, z = d == 2u ? far : b;
    li = x * 16u + y * 4u + z;
    // One step beyond the block: from the far end back across (4 cells) in the neighbour's frame.
    const uint32_t stride = d == 0u ? SOLVE_PX : d == 1u ? SOLVE_PY : 1u;
    at = solve_at(li) + (hi ? 4u * stride : 0u - 4u * stride);
}

// A lane's two cells of one block: the solver's values for them. `mask`: bits 0 and 1 whether the
// cells are water, 2 whether cell 0 has a water neighbour in the block, 4-6 and 8-10 how many of
// the cells' faces are not solid (the diagonal is a table of that count), 12-14 whether the lane's
// three cells across faces are water next to water. `zi`: those cells (or NONE);
// `hd` their search directions.
struct SolveCells {
    float z[2], d[2], r[2], p[2], q[2], dg[2], iv[2];
    uint32_t mask;
    uint32_t zi[3];
    float hd[3];
    __device__ __forceinline__ bool water(int k) const { return ((mask >> k) & 1u) != 0u; }
    __device__ __forceinline__ uint32_t faces(int k) const { return (mask >> (4 + 4 * k)) & 7u; }
};

// The record of a block whose warp has several: SolveCells by lane, without p (in F_P).
struct SolveRec {
    float2 z[32], d[32], r[32], q[32];
    float hd[3][32];
    uint32_t mask[32];
};
static_assert(sizeof(SolveRec) <= 64 * 32 && sizeof(SolveRec) % 16 == 0, "a block's record fits its part of D.wnb");
// Dynamic shared memory of a launch whose warps have several blocks: two CTAs an SM.
constexpr uint32_t SOLVE_DYN = 48u * sizeof(SolveRec);

// Shared memory by its own addresses.
__device__ __forceinline__ float lds_f(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_f(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }

// Symmetric red-black Gauss-Seidel, two sweeps inside the block (fluid.wgsl:390-410), by one
// warp. zl: the warp's padded array, -0 around the block: adding it leaves a sum as it is, its sign
// of zero too. The cells of one colour do not touch each other, so the order in which a half-sweep
// visits them does not matter. In the first half-sweep every neighbour is still +0.
__device__ __forceinline__ void warp_precondition(uint32_t zl, const SolveLane& L, SolveCells& C) {
    const bool w0 = C.water(0), w1 = C.water(1);
    sts_f(zl + 4u * L.at[1], w1 ? 0.0f : -0.0f);
    float z = div_by((C.mask & 4u) ? C.r[0] + 0.0f : C.r[0], C.dg[0], C.iv[0]);
    C.z[0] = z;
    sts_f(zl + 4u * L.at[0], w0 ? z : -0.0f);
    __syncwarp();
    auto sweep = [&](int k) {
        const uint32_t n = zl + 4u * L.at[k];
        const float a = lds_f(n - 4u * SOLVE_PX), b = lds_f(n + 4u * SOLVE_PX), c = lds_f(n - 4u * SOLVE_PY), d = lds_f(n + 4u * SOLVE_PY);
        const float e = lds_f(n - 4u), f = lds_f(n + 4u);
        z = div_by(((((((C.r[k] + a) + b) + c) + d) + e) + f), C.dg[k], C.iv[k]);
        sts_f(n, (k == 0 ? w0 : w1) ? z : -0.0f);
        C.z[k] = z;
        __syncwarp();
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
        sweep(1);
        sweep(0);
    }
    if (!w0) C.z[0] = 0.0f;
    if (!w1) C.z[1] = 0.0f;
}

// Where a CTA keeps its blocks' partial sums: its blocks are those of residues c, c + G,
// c + 2 G, ... (below 256), in that order and by ascending block within a residue; residue k's
// blocks are the CTA's E[k] .. E[k + 1] - 1. Quantity q of the CTA's e-th block, block b, is at
// part[q * stride + e] in shared memory, or part[q * stride + b] in the job's global array.
template <class A>
struct SolveParts {
    A* part;
    uint32_t stride;
    bool by_block;
    const uint32_t* E;
    uint32_t n_res;
    __device__ __forceinline__ A& at(uint32_t q, uint32_t e, uint32_t b) const { return part[q * stride + (by_block ? b : e)]; }
};

__device__ __forceinline__ uint32_t atom_add_release(uint32_t* p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Publishes this CTA's running sums (fluid.wgsl:429-431) of quantities 0..NQ-1 of `P`, waits at
// the grid barrier, and forms the 256-wide trees (fluid.wgsl:434-438): warp q quantity q's, lane l
// loading sums l, l + 32, ..., l + 224 (a residue without blocks, from nb on, is zero), the levels
// 128, 64 and 32 in registers and the rest with shuffles. Thread 0 then runs `post` on the trees,
// before a barrier: what it writes to shared memory every thread sees. The sums are double-buffered
// by the barrier's parity: a CTA writes the next-but-one sums only after every CTA has passed the
// next barrier, that is, has read these. False (in every thread) if the wait gave up.
template <class A, int NQ, class Post>
__device__ __forceinline__ bool exchange(const Dev& D, DevState* st, uint32_t& gen, const SolveParts<A>& P, uint32_t c, uint32_t G, uint32_t nb,
                                         Post&& post) {
    __shared__ uint32_t s_ok;
    __shared__ A s_out[SOLVE_XQ];
    gen++;
    double* sums = D.xsum + (size_t)(gen & 1u) * 256u * SOLVE_XQ;
    __syncthreads();  // every warp's partials and cell writes of this phase are done
    for (uint32_t t = threadIdx.x; t < P.n_res * NQ; t += blockDim.x) {
        const uint32_t k = t / NQ, q = t % NQ, r = c + k * G;
        const uint32_t e0 = P.E[k], e1 = P.E[k + 1];
        A s = A(0);
#pragma unroll 4
        for (uint32_t e = e0; e < e1; e++) s = s + P.at(q, e, r + 256u * (e - e0));
        if (e1 > e0) sums[q * 256u + r] = (double)s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // Release: this CTA's writes (ordered before by the barrier above) before the arrival.
        const uint32_t target = gen * G;
        if (!(gen == 1u && c == D.bar_skip)) atom_add_release(&st->bar_count, 1u);
        uint32_t ok = 1u;
        for (uint32_t spins = 0; ld_acquire(&st->bar_count) < target;) {
            // Give up after a bounded wait, or at once when another CTA of the solve has.
            if (++spins > D.bar_spins || ((spins & 1023u) == 0u && *(volatile uint32_t*)&st->err != 0u)) {
                atomicOr(&st->err, 1u);
                ok = 0u;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) return false;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (warp < (uint32_t)NQ) {
        A v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = lane + 32u * i < nb ? (A)__ldcg(sums + warp * 256u + lane + 32u * i) : A(0);
        // Level 128: positions l, l + 32, l + 64, l + 96 add l + 128, ... ; level 64; level 32.
        const A a0 = v[0] + v[4], a1 = v[1] + v[5], a2 = v[2] + v[6], a3 = v[3] + v[7];
        const A b0 = a0 + a2, b1 = a1 + a3;
        A x = b0 + b1;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, off);
        if (lane == 0) s_out[warp] = x;
        // Warp 0 takes the other quantities' trees.
        if (NQ > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * NQ) : "memory");
        if (threadIdx.x == 0) post(s_out);
    }
    __syncthreads();
    return true;
}

constexpr uint32_t SOLVE_MAX_JOBS = 128;  // systems solved by one launch, at most
constexpr uint32_t SOLVE_PART_SH = 256;   // partial sums per quantity kept in shared memory

// The CTAs of a launch split over its jobs (independent systems, each a simulation's step):
// every job that steps gets one CTA and the rest go by expected work, its blocks times its last
// solve's iterations, at most 256 each. Every CTA computes the same split. c0[j] .. c0[j + 1]
// are job j's CTAs. (A job's result does not depend on how many CTAs it gets.)
__device__ __forceinline__ void solve_split(const Dev* jobs, uint32_t n_jobs, uint32_t* w, uint32_t* c0) {
    for (uint32_t j = threadIdx.x; j < n_jobs; j += blockDim.x) {
        const DevState* st = jobs[j].st;
        w[j] = st->s.dt_ns == 0u ? NONE : min(st->s.n_blocks, jobs[j].cap_blocks) * max(min(st->iters_prev, 4096u), 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t live = 0;
        uint64_t total = 0;
        for (uint32_t j = 0; j < n_jobs; j++)
            if (w[j] != NONE) live++, total += w[j];
        const uint32_t spare = gridDim.x > live ? gridDim.x - live : 0u;
        uint32_t at = 0;
        for (uint32_t j = 0; j < n_jobs; j++) {
            c0[j] = at;
            if (w[j] == NONE || at >= gridDim.x) continue;
            const uint32_t extra = total ? (uint32_t)((uint64_t)spare * w[j] / total) : 0u;
            at += min(1u + extra, min(256u, gridDim.x - at));
        }
        c0[n_jobs] = at;
    }
    __syncthreads();
}

// The solve of one system by CTAs c = 0 .. G - 1 of a cooperative launch (k_solve for one
// simulation, k_solve_batch for several). A job's result does not depend on G: the sums are the
// reference's 256 running sums and tree either way. `recs`, `n_recs`: the CTA's dynamic shared
// memory, in records.
template <bool FP64>
__device__ __forceinline__ void solve_body(const Dev& D, uint32_t c, uint32_t G, SolveRec* recs, uint32_t n_recs) {
    using M = SolveMath<FP64>;
    using A = typename M::A;
    __shared__ uint32_t s_E[257];
    __shared__ A s_part[3 * SOLVE_PART_SH];
    __shared__ float s_zl[SOLVE_W][SOLVE_PAD], s_dl[SOLVE_W][SOLVE_PAD];
    __shared__ float s_diag[8], s_inv[8];
    DevState* st = D.st;
    if (st->s.dt_ns == 0) return;
    uint32_t gen = 0;
    const Grid g = grid_of(D, cur_of(st));
    const ntr_gpu_params* U = D.U;
    const uint32_t nb = min(st->s.n_blocks, D.cap_blocks);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SolveLane L((uint32_t)lane);
    const uint32_t zl = (uint32_t)__cvta_generic_to_shared(s_zl[warp]), dl = (uint32_t)__cvta_generic_to_shared(s_dl[warp]);
    uint32_t h_face[3], h_li[3], h_at[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        solve_halo((uint32_t)lane, (uint32_t)j, h_face[j], h_li[j], h_at[j]);
        sts_f(zl + 4u * h_at[j], -0.0f);
    }
    const float tol = U->solve[0];
    const uint32_t limit = U->limits[2];
    const float hh = g.h, dt = dt_of(st);
    const float rho = U->fluid[0];
    const float cs = U->gravity[3] * dt;
    const float kc = hh * hh / (cs * cs);
    const bool pushed = st->pushed != 0u;
    // Read before the first barrier: thread 0 of CTA 0 writes them back at the end. alpha keeps the last
    // step's value when the solver does not run, as the reference's state does.
    uint32_t iters_max = st->s.iters_max, unconverged = st->s.unconverged;
    double alpha = st->alpha;
    // This CTA's residues c, c + G, ... and their blocks.
    auto count_of = [&](uint32_t r) -> uint32_t { return r < nb ? (nb - r + 255u) / 256u : 0u; };
    const uint32_t n_res = c < 256u ? (256u - c + G - 1u) / G : 0u;
    if (threadIdx.x == 0) {
        uint32_t e = 0;
        for (uint32_t k = 0; k < n_res; k++) s_E[k] = e, e += count_of(c + k * G);
        s_E[n_res] = e;
        // The diagonal of a cell with n faces that are not solid: kc and n times 1 added in turn.
        float dg = kc;
        for (int n = 0; n < 8; n++) {
            s_diag[n] = dg, s_inv[n] = 1.0f / dg;
            dg += 1.0f;
        }
    }
    __syncthreads();
    const uint32_t n_mine = s_E[n_res];
    // The partial sums: in shared memory, or in the job's own array when the CTA has too many
    // blocks for that.
    SolveParts<A> P;
    P.by_block = n_mine > SOLVE_PART_SH;
    P.part = P.by_block ? reinterpret_cast<A*>(D.spart) : s_part;
    P.stride = P.by_block ? D.cap_blocks : SOLVE_PART_SH;
    P.E = s_E;
    P.n_res = n_res;
    // The CTA's e-th block: residue k (the last with E[k] <= e), its (e - E[k])-th block.
    auto block_of = [&](uint32_t e) -> uint32_t {
        uint32_t lo = 0, hi = n_res;  // E[lo] <= e < E[hi]
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) / 2u;
            if (s_E[mid] <= e) lo = mid; else hi = mid;
        }
        return c + lo * G + 256u * (e - s_E[lo]);
    };
    const uint32_t n_warp = n_mine > (uint32_t)warp ? (n_mine - 1u - (uint32_t)warp) / SOLVE_W + 1u : 0u;
    const bool in_regs = n_mine <= (uint32_t)SOLVE_W;
    const bool in_shared = n_mine <= n_recs;
    auto rec_of = [&](uint32_t e, uint32_t b) -> SolveRec* { return in_shared ? recs + e : reinterpret_cast<SolveRec*>(D.wnb + (size_t)b * 64u * 8u); };

    // The link of a face's neighbour block in block_nb.
    auto h_link = [](uint32_t f) -> uint32_t { return f == 0u ? 4u : f == 1u ? 22u : f == 2u ? 10u : f == 3u ? 16u : f == 4u ? 12u : 14u; };

    // ---- solve_init (fluid.wgsl:445-491): diagonal, right-hand side, residual, preconditioned
    // residual, and the block's (r.z, r.r, b.b).
    auto init_block = [&](SolveCells& C, uint32_t b, uint32_t e) {
        float bq[2];
        C.mask = 0u;
        uint32_t h_block[3];
#pragma unroll
        for (int j = 0; j < 3; j++) h_block[j] = g.nb[b * 27u + h_link(h_face[j])];
        // One cell after the other (to bound the registers), each with all its loads first.
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t cell = b * 64u + L.li[k];
            uint32_t nbr[6];
            float nty[6], np[6], nu[3], uc[3];
#pragma unroll
            for (int j = 0; j < 6; j++) nbr[j] = neighbour(g, cell, ed(j >> 1, (j & 1) ? 1 : -1));
            const float ty = cfv(D, F_TYPE, cell);
            const float pc = cfv(D, F_P, cell);
            const float dold = cfv(D, F_D, cell);
            const int32_t src = accv(D, A_SRC, cell);
#pragma unroll
            for (int d = 0; d < 3; d++) uc[d] = face_pushed(D, d, cell, pushed);
#pragma unroll
            for (int j = 0; j < 6; j++) {
                nty[j] = GAS_T, np[j] = 0.0f;
                if (nbr[j] != NONE) nty[j] = cfv(D, F_TYPE, nbr[j]), np[j] = cfv(D, F_P, nbr[j]);
            }
#pragma unroll
            for (int d = 0; d < 3; d++) nu[d] = nbr[2 * d + 1] != NONE ? face_pushed(D, d, nbr[2 * d + 1], pushed) : 0.0f;
            const bool water = ty == WATER_T;
            sts_f(dl + 4u * L.at[k], water ? 1.0f : 0.0f);  // for the masks below
            C.r[k] = 0.0f, C.p[k] = pc, C.d[k] = water ? dold : 0.0f, C.q[k] = 0.0f, C.z[k] = 0.0f, bq[k] = 0.0f;
            if (!water) continue;
            uint32_t n_face = 0u;
            bool inside = false;  // a water neighbour in the block
            float div = 0.0f, off = 0.0f;
            float bb = kc * pc;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                // face_u of the face above (its cell the neighbour, below it this cell) minus
                // the face below (this cell over the neighbour below).
                const float fu_hi = nbr[2 * d + 1] == NONE ? 0.0f : bounded(nu[d], nty[2 * d + 1], ty);
                const float fu_lo = bounded(uc[d], ty, nty[2 * d]);
                div += fu_hi - fu_lo;
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    const int j = 2 * d + s;
                    if (nty[j] == SOLID_T) continue;
                    n_face++;
                    if (nty[j] == WATER_T) {
                        off -= np[j];
                        inside = inside || (nbr[j] >> 6) == b;
                    } else {
                        bb += np[j];  // pressure_of: 0 outside the grid, p of a non-water cell
                    }
                }
            }
            const float dg = s_diag[n_face];
            div -= from_fp(src, FP_Q) / (hh * hh);
            bb -= rho * hh / dt * div;
            C.r[k] = bb - dg * pc - off;
            bq[k] = bb;
            C.mask |= (1u << k) | (k == 0 && inside ? 4u : 0u) | (n_face << (4 + 4 * k));
            *cfp(D, F_DIAG, cell) = dg;
            *cfp(D, F_R, cell) = C.r[k];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint32_t s = h_face[j] < 2u ? SOLVE_PX : h_face[j] < 4u ? SOLVE_PY : 1u;
            // A cell across a face counts when it and the block's cell next to it are water.
            const bool own = lds_f(dl + 4u * ((h_face[j] & 1u) ? h_at[j] - s : h_at[j] + s)) != 0.0f;
            C.hd[j] = 0.0f, C.zi[j] = NONE;
            if (own && h_block[j] != NONE && cfv(D, F_TYPE, h_block[j] * 64u + h_li[j]) == WATER_T) {
                C.hd[j] = cfv(D, F_D, h_block[j] * 64u + h_li[j]);
                C.zi[j] = h_block[j] * 64u + h_li[j];
                C.mask |= 1u << (12 + j);
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 2; k++) C.dg[k] = s_diag[C.faces(k)], C.iv[k] = s_inv[C.faces(k)];
        warp_precondition(zl, L, C);
        for (int k = 0; k < 2; k++)
            if (C.water(k)) *cfp(D, F_Z, b * 64u + L.li[k]) = C.z[k];
        A sz = warp_tree64(L, M::prod(bq[0], bq[0]), M::prod(bq[1], bq[1]));
        A sxy = warp_tree64x2(L, (uint32_t)lane, M::prod(C.r[0], C.z[0]), M::prod(C.r[1], C.z[1]), M::prod(C.r[0], C.r[0]), M::prod(C.r[1], C.r[1]));
        if (lane == 0) P.at(0, e, b) = sxy, P.at(2, e, b) = sz;
        if (lane == 16) P.at(1, e, b) = sxy;
    };

    // The residuals across the block's faces, written by other warps and CTAs earlier in this
    // launch: read through L2.
    auto load_hz = [&](const SolveCells& C, float (&hz)[3]) {
#pragma unroll
        for (int j = 0; j < 3; j++) hz[j] = C.zi[j] != NONE ? __ldcg(cfp(D, F_Z, C.zi[j])) : 0.0f;
    };

    // ---- solve_q (fluid.wgsl:513-534): the new search direction and A d. `hz`: load_hz's.
    auto q_block = [&](SolveCells& C, uint32_t b, uint32_t e, float fbeta, const float (&hz)[3]) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            if (C.zi[j] != NONE) C.hd[j] = hz[j] + fbeta * C.hd[j];
            sts_f(dl + 4u * h_at[j], C.hd[j]);
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (C.water(k)) C.d[k] = C.z[k] + fbeta * C.d[k];
            sts_f(dl + 4u * L.at[k], C.d[k]);  // +0 where not water
        }
        __syncwarp();
        A v[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t n = dl + 4u * L.at[k];
            const float a = lds_f(n - 4u * SOLVE_PX), b = lds_f(n + 4u * SOLVE_PX), c = lds_f(n - 4u * SOLVE_PY), d = lds_f(n + 4u * SOLVE_PY);
            const float e = lds_f(n - 4u), f = lds_f(n + 4u);
            const float q = ((((((C.dg[k] * C.d[k]) - a) - b) - c) - d) - e) - f;
            C.q[k] = q;
            v[k] = C.water(k) ? M::prod(C.d[k], q) : A(0);
        }
        const A s = warp_tree64(L, v[0], v[1]);
        if (lane == 0) P.at(0, e, b) = s;
        __syncwarp();
    };

    // ---- solve_update (fluid.wgsl:543-559): p, r, and the preconditioned residual.
    auto update_block = [&](SolveCells& C, uint32_t b, uint32_t e, float a) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (!C.water(k)) continue;
            C.p[k] = C.p[k] + a * C.d[k];
            C.r[k] = C.r[k] - a * C.q[k];
        }
        warp_precondition(zl, L, C);
#pragma unroll
        for (int k = 0; k < 2; k++)
            if (C.water(k)) *cfp(D, F_Z, b * 64u + L.li[k]) = C.z[k];
        const A s = warp_tree64x2(L, (uint32_t)lane, M::prod(C.r[0], C.z[0]), M::prod(C.r[1], C.z[1]), M::prod(C.r[0], C.r[0]), M::prod(C.r[1], C.r[1]));
        if (lane == 0) P.at(0, e, b) = s;
        if (lane == 16) P.at(1, e, b) = s;
    };

    // The record of one of a warp's several blocks: what a phase needs of it.
    auto load_rec = [&](SolveCells& C, const SolveRec* R, uint32_t b) {
        const float2 z = R->z[lane], d = R->d[lane], r = R->r[lane], q = R->q[lane];
        C.z[0] = z.x, C.z[1] = z.y, C.d[0] = d.x, C.d[1] = d.y, C.r[0] = r.x, C.r[1] = r.y, C.q[0] = q.x, C.q[1] = q.y;
        C.mask = R->mask[lane];
#pragma unroll
        for (int k = 0; k < 2; k++) C.dg[k] = s_diag[C.faces(k)], C.iv[k] = s_inv[C.faces(k)];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            C.zi[j] = ((C.mask >> (12 + j)) & 1u) ? g.nb[b * 27u + h_link(h_face[j])] * 64u + h_li[j] : NONE;
            C.hd[j] = R->hd[j][lane];
        }
    };

    SolveCells C;
    float hz[3];
    const uint32_t b_reg = n_warp ? block_of((uint32_t)warp) : 0u;  // the block of a warp with one
    if (in_regs) {
        if (n_warp) init_block(C, b_reg, (uint32_t)warp);
    } else {
        for (uint32_t j = 0; j < n_warp; j++) {
            const uint32_t e = (uint32_t)warp + j * SOLVE_W, b = block_of(e);
            SolveRec* R = rec_of(e, b);
            init_block(C, b, e);
            R->z[lane] = make_float2(C.z[0], C.z[1]), R->d[lane] = make_float2(C.d[0], C.d[1]);
            R->r[lane] = make_float2(C.r[0], C.r[1]), R->q[lane] = make_float2(0.0f, 0.0f);
            R->mask[lane] = C.mask;
#pragma unroll
            for (int k = 0; k < 3; k++) R->hd[k][lane] = C.hd[k];
        }
        __syncwarp();
    }

    // The scalars of the iteration are thread 0's; the others get what they need of them.
    __shared__ float s_scalar;
    __shared__ bool s_on;

    // solve_start (fluid.wgsl:493-506).
    double rz = 0.0, beta = 0.0, b_norm = 0.0, r_norm = 0.0;
    uint32_t iters = 0;
    if (!exchange<A, 3>(D, st, gen, P, c, G, nb, [&](const A* s) {
            rz = (double)s[0];
            b_norm = M::root((double)s[2]);
            r_norm = M::root((double)s[1]);
            s_on = (double)s[0] > 0.0 && !M::converged((double)s[1], b_norm, tol);
            s_scalar = 0.0f;
        }))
        return;
    while (s_on) {
        const float fbeta = s_scalar;
        if (in_regs) {
            if (n_warp) {
                load_hz(C, hz);
                q_block(C, b_reg, (uint32_t)warp, fbeta, hz);
            }
        } else {
            for (uint32_t j = 0; j < n_warp; j++) {
                const uint32_t e = (uint32_t)warp + j * SOLVE_W, b = block_of(e);
                SolveRec* R = rec_of(e, b);
                load_rec(C, R, b);
                load_hz(C, hz);
                q_block(C, b, e, fbeta, hz);
                R->d[lane] = make_float2(C.d[0], C.d[1]), R->q[lane] = make_float2(C.q[0], C.q[1]);
#pragma unroll
                for (int k = 0; k < 3; k++) R->hd[k][lane] = C.hd[k];
            }
        }
        // solve_alpha (fluid.wgsl:536-541).
        if (!exchange<A, 1>(D, st, gen, P, c, G, nb, [&](const A* s) {
                alpha = (double)s[0] > 0.0 ? M::ratio(rz, (double)s[0]) : 0.0;
                s_scalar = (float)alpha;
            }))
            return;
        const float a = s_scalar;
        if (in_regs) {
            if (n_warp) update_block(C, b_reg, (uint32_t)warp, a);
        } else {
            for (uint32_t j = 0; j < n_warp; j++) {
                const uint32_t e = (uint32_t)warp + j * SOLVE_W, b = block_of(e);
                SolveRec* R = rec_of(e, b);
                for (int k = 0; k < 2; k++) C.p[k] = cfv(D, F_P, b * 64u + L.li[k]);
                load_rec(C, R, b);
                update_block(C, b, e, a);
                R->z[lane] = make_float2(C.z[0], C.z[1]), R->r[lane] = make_float2(C.r[0], C.r[1]);
                for (int k = 0; k < 2; k++)
                    if (C.water(k)) *cfp(D, F_P, b * 64u + L.li[k]) = C.p[k];
            }
        }
        iters++;
        // solve_beta (fluid.wgsl:561-578).
        if (!exchange<A, 2>(D, st, gen, P, c, G, nb, [&](const A* s) {
                r_norm = M::root((double)s[1]);
                beta = rz > 0.0 ? M::ratio((double)s[0], rz) : 0.0;
                rz = (double)s[0];
                const bool done = M::converged((double)s[1], b_norm, tol);
                s_on = !(done || iters >= limit);
                s_scalar = (float)beta;
                if (!s_on) {
                    iters_max = max(iters_max, iters);
                    unconverged += done ? 0u : 1u;
                }
            }))
            return;
    }
    // What was kept on the chip goes to memory once, as the iterations would have left it.
    if (iters > 0)
        for (uint32_t j = 0; j < n_warp; j++) {
            const uint32_t e = (uint32_t)warp + j * SOLVE_W, b = block_of(e);
            if (!in_regs) load_rec(C, rec_of(e, b), b);
            for (int k = 0; k < 2; k++) {
                if (!C.water(k)) continue;
                const uint32_t cell = b * 64u + L.li[k];
                if (in_regs) *cfp(D, F_P, cell) = C.p[k];
                *cfp(D, F_R, cell) = C.r[k];
                *cfp(D, F_Q, cell) = C.q[k];
            }
        }
    if (c == 0 && threadIdx.x == 0) {
        st->rz = rz, st->alpha = alpha, st->beta = beta, st->b_norm = b_norm, st->r_norm = r_norm;
        st->solver_on = 0u;
        st->s.solve_iters = iters, st->s.iters_max = iters_max, st->s.unconverged = unconverged;
        st->s.rz = (float)rz, st->s.alpha = (float)alpha, st->s.beta = (float)beta;
        st->s.b_norm = (float)b_norm, st->s.r_norm = (float)r_norm;
    }
}

// The dynamic shared memory of a launch, in block records.
__device__ __forceinline__ SolveRec* solve_recs(uint32_t& n) {
    extern __shared__ __align__(16) uint8_t s_dyn[];
    uint32_t bytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(bytes));
    n = bytes / (uint32_t)sizeof(SolveRec);
    return reinterpret_cast<SolveRec*>(s_dyn);
}

template <bool FP64>
__global__ void __launch_bounds__(SOLVE_T, 2) k_solve(Dev D) {
    uint32_t n_recs;
    SolveRec* recs = solve_recs(n_recs);
    solve_body<FP64>(D, blockIdx.x, gridDim.x, recs, n_recs);
}

// One launch for the systems of `n_jobs` simulations (their pointer tables at `jobs`): the CTAs
// split over them (solve_split) and each group solves its own.
template <bool FP64>
__global__ void __launch_bounds__(SOLVE_T, 2) k_solve_batch(const Dev* __restrict__ jobs, uint32_t n_jobs) {
    __shared__ uint32_t s_w[SOLVE_MAX_JOBS], s_c0[SOLVE_MAX_JOBS + 1];
    __shared__ Dev s_dev;
    solve_split(jobs, n_jobs, s_w, s_c0);
    uint32_t job = NONE;
    for (uint32_t j = 0; j < n_jobs; j++)
        if (blockIdx.x >= s_c0[j] && blockIdx.x < s_c0[j + 1]) job = j;
    if (job == NONE) return;
    for (uint32_t k = threadIdx.x; k < sizeof(Dev) / 4; k += blockDim.x)
        reinterpret_cast<uint32_t*>(&s_dev)[k] = reinterpret_cast<const uint32_t*>(jobs + job)[k];
    __syncthreads();
    uint32_t n_recs;
    SolveRec* recs = solve_recs(n_recs);
    solve_body<FP64>(s_dev, blockIdx.x - s_c0[job], s_c0[job + 1] - s_c0[job], recs, n_recs);
}

}  // namespace ntr
