// EBE matvec and the batched restarted GMRES engine (sm_103a).
//
// Method (00_CommonFiles/Solvers_and_Preconditioners/pgmres.c:5-200):
// restarted, left-preconditioned GMRES(kmax) with X0 = 0, at most kmax-1
// Arnoldi steps per cycle (pgmres.c:159), Givens rotations (:120-155),
// back-substitution (:163-171) and X += V y (:173-175).  The reference's
// modified Gram-Schmidt with one MPI_Allreduce per dot becomes classical
// Gram-Schmidt with a Gram correction (the second classical pass' coefficients
// from the basis' Gram matrix): two streaming passes over the basis per step,
// each ending in a deterministic device-wide reduction (fixed part order, "last
// part reduces"), instead of 2(i+1) dependent reductions; batches that fit it
// run their cycles on chip (cycle.cu).
//
// Work decomposition.  A batch holds any number of systems.  The operator
// is the assembled one (rows.cu), cut into unit chunks, dof work into parts
// per system; every kernel walks its chunk table with a grid-stride loop and skips systems
// that are not active.  A system's sums depend on its own parts and gang only.
// In a batch of fewer than kSoloDofs equations these are the ones that the system
// has alone, so that a result has the same bits alone and in the batch; in a
// larger one part sizes, gangs and the engine follow the batch (and who has
// stopped), and results agree to rounding.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <type_traits>

#include <cuda_fp16.h>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "sums.cuh"

namespace fg {

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T> __device__ __forceinline__ T ldst(const T *p) { return __ldcs(p); }


// Last-part election: returns true in the CTA that completed the final part
// of system D (`split` CTAs a part) for counter slot `slot` (all threads of the
// CTA agree).
__device__ __forceinline__ bool last_part(const SysDev &D, int slot, unsigned split = 1)
{
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned prev = atomicAdd(&D.counter[slot], 1u);
        s_last = (prev == split * (unsigned)D.nparts - 1u);
        if (s_last) D.counter[slot] = 0u;
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Deterministic sum over parts of slots [0, nv), nv <= kPartStride: thread
// (sub, slot) adds parts sub, sub + S, ... in order (consecutive slots are
// consecutive addresses; the fewest FP64 instructions), then the S subs in
// order.  Results to out[] (shared).
__device__ __forceinline__ void reduce_parts(const SysDev &D, int nv, double *out)
{
    __shared__ double sub_sum[kThreads];
    const int L = nv <= 4 ? 4 : nv <= 64 ? 64 : kPartStride, S = kThreads / L;
    const int slot = threadIdx.x % L, sub = threadIdx.x / L;
    double s = 0.0;
    if (slot < nv) {
        const double *p = D.part + slot;
        int q = sub;
        for (; q + 3 * S < D.nparts; q += 4 * S) {
            const double a = __ldcg(p + (size_t)q * kPartStride), b = __ldcg(p + (size_t)(q + S) * kPartStride);
            const double c = __ldcg(p + (size_t)(q + 2 * S) * kPartStride), d = __ldcg(p + (size_t)(q + 3 * S) * kPartStride);
            s += (a + b) + (c + d);
        }
        for (; q < D.nparts; q += S) s += __ldcg(p + (size_t)q * kPartStride);
    }
    sub_sum[threadIdx.x] = s;
    __syncthreads();
    for (int w = S / 2; w >= 1; w >>= 1) {
        if (sub < w) sub_sum[threadIdx.x] += sub_sum[threadIdx.x + w * L];
        __syncthreads();
    }
    if (threadIdx.x < nv) out[threadIdx.x] = sub_sum[threadIdx.x];
    __syncthreads();
}

// ---------------------------------------------------------------- EBE matvec
// y[lm] += A_e x[lm] by patches.  A patch is up to patch_elems(S)
// consecutive elements (internal order: sorted by their smallest dof, so a
// patch covers a compact band of dofs).  The CTAs loop over the patches of
// their launch (one launch per patch colour); per patch:
//  1. x of the patch's dofs is gathered into shared memory;
//  2. the element products A_e x_e are formed and staged in shared memory
//     with the elements' local indices, one thread per element; A and lm16 are
//     SoA [entry][element], so lane-consecutive elements read consecutive
//     addresses;
//  3. the staged rows are added into a shared-memory y local colour by local
//     colour (elements of one local colour share no dof: no atomics, a fixed
//     summation order), then each dof is written once: a plain store for
//     dofs only this patch touches, a reduction store (red.add) for dofs
//     shared with other patches (patches sharing a dof have different patch
//     colours and run in different launches, so the updates apply in launch
//     order, as read-modify-writes would).
// (3x3 blocks: k_ebe_mv3.)
// The patch sizes (patch_elems) and this kernel shape were chosen by a
// measured sweep: an L2 prefetch of the next patch, one thread per block
// row with small patches, and a two-stage copy pipeline through shared
// memory were all slower.  The sink (index n) is never written.
// x and y are FP64; fg_matvec and fg_matvec_noalloc use these (the Krylov engine
// has the assembled operator, rows.cu).
template <int S, typename TA>
__global__ void __launch_bounds__(kThreads, sizeof(TA) == 4 ? 4 : 3)
k_ebe_mv(const SysDev *__restrict__ sys, const EChunk *__restrict__ ch, const int *__restrict__ nch,
         const double *__restrict__ X, double *Y, int maxdof)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned short kSink = 0xFFFF;
    constexpr int PE = patch_elems(S);
    const MvSmem L(S, maxdof, (int)sizeof(TA));
    TA *xs = reinterpret_cast<TA *>(smem_raw + L.xs);
    TA *ys = reinterpret_cast<TA *>(smem_raw + L.ys);
    TA *ye = reinterpret_cast<TA *>(smem_raw + L.ye);
    unsigned short *ls = reinterpret_cast<unsigned short *>(smem_raw + L.ls);
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const EChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        const TA *A = sizeof(TA) == 8 ? (const TA *)D.A64 : (const TA *)D.A32;
        const size_t ld = (size_t)D.nel_pad;
        const int p = k.e0;
        const int pe0 = D.pt_elem[p], pne = D.pt_elem[p + 1] - pe0;
        const int pd0 = D.pt_dof[p], pnd = D.pt_dof[p + 1] - pd0;
        const unsigned short *pc = D.pt_col + (size_t)p * kPatchColStride;
        __syncthreads();                      // the previous patch is done with shared memory
        for (int j = threadIdx.x; j < pnd; j += kThreads) {
            xs[j] = (TA)X[D.dofs[pd0 + j] & 0x7fffffff];
            ys[j] = (TA)0;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < pne; q += kThreads) {
            unsigned short l[S];
            TA xv[S];
#pragma unroll
            for (int a = 0; a < S; ++a) {
                l[a] = __ldcs(D.lm16 + a * ld + pe0 + q);
                xv[a] = l[a] == kSink ? (TA)0 : xs[l[a]];
            }
#pragma unroll
            for (int r = 0; r < S; ++r) {
                TA acc = ldst(A + (size_t)(r * S) * ld + pe0 + q) * xv[0];
#pragma unroll
                for (int m = 1; m < S; ++m) acc += ldst(A + (size_t)(r * S + m) * ld + pe0 + q) * xv[m];
                ye[r * PE + q] = acc;
                ls[r * PE + q] = l[r];
            }
        }
        __syncthreads();
        for (int col = 0; col < kPatchMaxLocalColours; ++col) {
            const int cs = pc[col], ce = pc[col + 1];
            if (cs >= ce) break;
            for (int q = cs + threadIdx.x; q < ce; q += kThreads) {
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const unsigned short l = ls[r * PE + q];
                    if (l != kSink) ys[l] += ye[r * PE + q];
                }
            }
            __syncthreads();
        }
        // a dof shared with other patches takes a reduction store (no round
        // trip); the patches of one launch share no dof, so each update is
        // Y[d] + v in launch order, as a read-modify-write would be
        for (int j = threadIdx.x; j < pnd; j += kThreads) {
            const int dd = D.dofs[pd0 + j];
            const int d = dd & 0x7fffffff;
            if (d == D.n) continue;                       // dof-list padding
            if (dd < 0) atomicAdd(Y + d, (double)ys[j]);
            else Y[d] = (double)ys[j];
        }
    }
}

// The FP64 S x S matvec (S = 6, 9, 12) with a thread per (element, block
// row) pair of the patch instead of a thread per element, in CTAs of 512
// threads.  A patch colour of a mesh in natural node order holds only a
// few hundred patches (7 colours of 256-element patches on a structured
// mesh), so one launch has that many CTAs: per-element threads left 20% of
// the warp slots filled, the FP64 pipe 40% busy and the loads of A waiting
// on each other (ncu: long-scoreboard stalls); per-pair threads put S
// times more independent rows in flight per CTA (12x12: 1.75 -> 2.07 TB/s
// at 385x385).  In FP32 the S-fold x gathers from shared memory cost more
// than that gains (9x9: 2.70 -> 1.97 TB/s), so FP32 keeps k_ebe_mv.  Per patch: x gathered and the patch's local
// indices staged in shared memory; each pair forms its row product exactly
// as the per-element kernel does (acc = A_r0 x_0, then acc += A_rm x_m in
// m order) and stages it; the staged rows are added into the shared y
// local colour by local colour; each dof is written once (plain store, or
// red.add for a dof shared with patches of other colours).  Same sums in
// the same order as k_ebe_mv, so the results are bit-identical.
constexpr int kMvbThreads = 512;
// rows per thread: FP64 one (every warp slot for the FP64 pipe); FP32 S /
// FG_MVB_GROUPS32 row groups per element, 0 (the default) the per-element
// k_ebe_mv: measured in FP32 (Euler 385^2 12x12 / NS 513^2 9x9, TB/s),
// per element 1.82 / 2.70, one group of 512-thread CTAs 1.87 / 1.92, three
// row groups 1.82 / 2.15.
#ifndef FG_MVB_GROUPS32
#define FG_MVB_GROUPS32 0
#endif
template <int S, typename TA> constexpr int mvb_rows()
{
    constexpr int g = FG_MVB_GROUPS32 > 0 ? FG_MVB_GROUPS32 : 1;
    return sizeof(TA) == 8 ? 1 : (FG_MVB_GROUPS32 > 0 && S > 3 && S % g == 0) ? S / g : 0;
}
template <int S, typename TA>
__global__ void __launch_bounds__(kMvbThreads, 2)
k_ebe_mvb(const SysDev *__restrict__ sys, const EChunk *__restrict__ ch, const int *__restrict__ nch,
          const double *__restrict__ X, double *Y, int maxdof)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned short kSink = 0xFFFF;
    constexpr int PE = patch_elems(S);
    const MvSmem L(S, maxdof, (int)sizeof(TA));
    TA *xs = reinterpret_cast<TA *>(smem_raw + L.xs);
    TA *ys = reinterpret_cast<TA *>(smem_raw + L.ys);
    TA *ye = reinterpret_cast<TA *>(smem_raw + L.ye);
    unsigned short *ls = reinterpret_cast<unsigned short *>(smem_raw + L.ls);
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const EChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        const TA *A = sizeof(TA) == 8 ? (const TA *)D.A64 : (const TA *)D.A32;
        const size_t ld = (size_t)D.nel_pad;
        const int p = k.e0;
        const int pe0 = D.pt_elem[p], pne = D.pt_elem[p + 1] - pe0;
        const int pd0 = D.pt_dof[p], pnd = D.pt_dof[p + 1] - pd0;
        const unsigned short *pc = D.pt_col + (size_t)p * kPatchColStride;
        __syncthreads();                      // the previous patch is done with shared memory
        for (int j = threadIdx.x; j < pnd; j += kMvbThreads) {
            xs[j] = (TA)X[D.dofs[pd0 + j] & 0x7fffffff];
            ys[j] = (TA)0;
        }
        for (int e = threadIdx.x; e < S * pne; e += kMvbThreads) {
            const int a = e / pne, q = e - a * pne;
            ls[a * PE + q] = __ldcs(D.lm16 + a * ld + pe0 + q);
        }
        __syncthreads();
        constexpr int R = mvb_rows<S, TA>() > 0 ? mvb_rows<S, TA>() : 1, NG = S / R;
        static_assert(S % R == 0, "rows per thread must divide the block");
        for (int e = threadIdx.x; e < NG * pne; e += kMvbThreads) {
            const int g = e / pne, q = e - g * pne;
            TA xv[S];
#pragma unroll
            for (int a = 0; a < S; ++a) {
                const unsigned short l = ls[a * PE + q];
                xv[a] = l == kSink ? (TA)0 : xs[l];
            }
#pragma unroll
            for (int rr = 0; rr < R; ++rr) {
                const int r = g * R + rr;
                const TA *Ar = A + (size_t)(r * S) * ld + pe0 + q;
                TA acc = ldst(Ar) * xv[0];
#pragma unroll
                for (int m = 1; m < S; ++m) acc += ldst(Ar + (size_t)m * ld) * xv[m];
                ye[r * PE + q] = acc;
            }
        }
        __syncthreads();
        for (int col = 0; col < kPatchMaxLocalColours; ++col) {
            const int cs = pc[col], ce = pc[col + 1];
            if (cs >= ce) break;
            for (int q = cs + threadIdx.x; q < ce; q += kMvbThreads) {
#pragma unroll
                for (int r = 0; r < S; ++r) {
                    const unsigned short l = ls[r * PE + q];
                    if (l != kSink) ys[l] += ye[r * PE + q];
                }
            }
            __syncthreads();
        }
        for (int j = threadIdx.x; j < pnd; j += kMvbThreads) {
            const int dd = D.dofs[pd0 + j];
            const int d = dd & 0x7fffffff;
            if (d == D.n) continue;                       // dof-list padding
            if (dd < 0) atomicAdd(Y + d, (double)ys[j]);
            else Y[d] = (double)ys[j];
        }
    }
}

// 16-byte asynchronous copy global -> shared (cp.async, L2 only) and its wait.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// The 3x3 matvec: per patch, the dof list, element blocks and local
// indices are loaded into registers (one round trip), x of the patch's dofs
// is gathered into shared memory while the patch's incidence lists arrive
// there by asynchronous copies, the element products are staged in shared
// memory, and then the thread that gathered a dof sums the products that add
// into it, in the fixed order of its incidence list, and writes it: a plain
// store for a dof only this patch touches, a reduction store (red.add) for
// one shared with other patches (those run in other launches, so the updates
// apply in launch order).  Two barriers per patch; every thread sums whole
// dofs, so no shared-memory y and no colour passes.
template <typename TA>
// FP32: 64 registers, 4 CTAs per SM (56 bytes of spills; measured 3.78 vs
// 3.72 TB/s at 80 registers and 3 CTAs)
__global__ void __launch_bounds__(kThreads, sizeof(TA) == 4 ? 4 : 2)
k_ebe_mv3(const SysDev *__restrict__ sys, const EChunk *__restrict__ ch, const int *__restrict__ nch,
          const double *__restrict__ X, double *Y, int maxdof)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr unsigned short kSink = 0xFFFF;
    constexpr int PE = patch_elems(3);
    constexpr int E = PE / kThreads;        // elements per thread
    constexpr int DMAX = 1536 / kThreads;   // patch dofs per thread (the patch cap)
    const MvSmem L(3, maxdof, (int)sizeof(TA));
    TA *xs = reinterpret_cast<TA *>(smem_raw + L.xs);
    TA *ye = reinterpret_cast<TA *>(smem_raw + L.ye);
    unsigned short *ic = reinterpret_cast<unsigned short *>(smem_raw + L.ic);
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const EChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        const TA *A = sizeof(TA) == 8 ? (const TA *)D.A64 : (const TA *)D.A32;
        const size_t ld = (size_t)D.nel_pad;
        const int p = k.e0;
        const int pe0 = D.pt_elem[p], pne = D.pt_elem[p + 1] - pe0;
        const int pd0 = D.pt_dof[p], pnd = D.pt_dof[p + 1] - pd0;
        const int i0 = D.pt_inc[p], ni = D.pt_inc[p + 1] - i0;
        const int head = (pnd + 1 + 7) & ~7;
        const int W = (pne + 15) & ~15;       // staged product row (FP32 blocks: blocked row) length
        // FP64 blocks are [entry][element]; FP32 blocks of a patch are one
        // block [entry][W] at 9 pe0
        const TA *Ap = sizeof(TA) == 8 ? A + pe0 : A + 9 * (size_t)pe0;
        const size_t lda = sizeof(TA) == 8 ? ld : (size_t)W;
        int dv[DMAX];
#pragma unroll
        for (int u = 0; u < DMAX; ++u) {
            const int j = threadIdx.x + u * kThreads;
            dv[u] = j < pnd ? __ldg(D.dofs + pd0 + j) : 0;
        }
        TA av[E][9];
        unsigned short li[E][3];
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int q = min(threadIdx.x + u * kThreads, pne - 1);
#pragma unroll
            for (int a = 0; a < 3; ++a) li[u][a] = __ldcs(D.lm16 + a * ld + pe0 + q);
#pragma unroll
            for (int m = 0; m < 9; ++m) av[u][m] = ldst(Ap + m * lda + q);
        }
        __syncthreads();                      // the previous patch is done with shared memory
        for (int t = threadIdx.x; t < ni / 8; t += kThreads) cp_async16(ic + 8 * t, D.incl + i0 + 8 * t);
#pragma unroll
        for (int u = 0; u < DMAX; ++u) {
            const int j = threadIdx.x + u * kThreads;
            if (j < pnd) xs[j] = (TA)X[dv[u] & 0x7fffffff];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int q = threadIdx.x + u * kThreads;
            if (q >= pne) continue;
            TA xv[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) xv[a] = li[u][a] == kSink ? (TA)0 : xs[li[u][a]];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                TA acc = av[u][3 * r] * xv[0];
                acc += av[u][3 * r + 1] * xv[1];
                acc += av[u][3 * r + 2] * xv[2];
                ye[r * W + q] = acc;
            }
        }
        cp_async_wait_all();
        __syncthreads();
#pragma unroll
        for (int u = 0; u < DMAX; ++u) {
            const int j = threadIdx.x + u * kThreads;
            const int dd = dv[u];
            const int d = dd & 0x7fffffff;
            if (j >= pnd || d == D.n) continue;           // dof-list padding
            const int e0 = ic[j], e1 = ic[j + 1];
            TA v = (TA)0;
            for (int e = e0; e < e1; ++e) v += ye[ic[head + e]];
            if (dd < 0) atomicAdd(Y + d, (double)v);          // shared dof: reduction store
            else Y[d] = (double)v;
        }
    }
}

// ---------------------------------------------------------------- CSR SpMV
// y = A x for the assembled operator (csrmv.c:57-62), W lanes per row
// (W = 4, 8 or 32 from the mean row length; rows of P1 transport hold ~7
// entries, rows of the 4-dof Euler system ~30): lanes stride the row,
// shuffle-reduce, one lane stores.  Works on dof parts like the Krylov
// kernels (fg_matvec; solves use the assembled blocks, rows.cu).
template <int W, typename TA>
__global__ void __launch_bounds__(kThreads)
k_csr_mv(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch,
         const double *__restrict__ X, double *Y)
{
    const int total = *nch;
    const int sub = threadIdx.x % W, grp = threadIdx.x / W, ngrp = blockDim.x / W;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        const TA *AA = sizeof(TA) == 8 ? (const TA *)D.AA64 : (const TA *)D.AA32;
        for (int base = k.d0; base < k.d1; base += ngrp) {
            const int row = base + grp;
            TA s = 0;
            if (row < k.d1)
                for (int q = D.csr_ia[row] + sub; q < D.csr_ia[row + 1]; q += W)
                    s += ldst(AA + q) * (TA)X[__ldcs(D.csr_ja + q)];
#pragma unroll
            for (int o = W / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, W);
            if (row < k.d1 && sub == 0) Y[row] = (double)s;
        }
    }
}

// ---------------------------------------------------------------- block-diagonal apply
// z[dofs of node] = invB(node) * p[dofs of node] (BlockDiag_precond.c:3-29,
// BlockDiagDOF3_precond.c:3-27); dofs that are Dirichlet read 0 and are not
// written.  The cycle start's t64 -> u64; in the Arnoldi steps the matvec
// applies it (rows.cu).
template <int B>
__global__ void __launch_bounds__(kThreads)
k_blockdiag(const SysDev *__restrict__ sys, const NChunk *__restrict__ ch, const int *__restrict__ nch)
{
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const NChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->live) continue;
        for (int nd = k.n0 + threadIdx.x; nd < k.n1; nd += blockDim.x) {
            int id[B];
            double v[B];
#pragma unroll
            for (int a = 0; a < B; ++a) {
                id[a] = D.node_dof[nd * B + a];
                v[a] = id[a] == D.n ? 0.0 : D.t64[id[a]];
            }
            const double *m = D.ibd64 + (size_t)nd * B * B;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                double s = m[r * B] * v[0];
#pragma unroll
                for (int q = 1; q < B; ++q) s += m[r * B + q] * v[q];
                if (id[r] != D.n) D.u64[id[r]] = s;
            }
        }
    }
}

// ---------------------------------------------------------------- cycle start
// FP64: u = M^-1 (A x) (t64 holds A x; for the block-diagonal case u64
// already holds M^-1 t64), r = b - u (pgmres.c:64-75), partial ||r||^2,
// true residual s = F - A x, partial ||s||^2, and on the first cycle ||b||^2
// and ||F||^2.
__global__ void __launch_bounds__(kThreads)
k_start(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch)
{
    __shared__ double red[4][kThreads / 32];
    __shared__ double tot[4];
    const int total = *nch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->live) continue;
        const bool first = D.st->first != 0;
        const bool has_f = D.ftrue != nullptr;
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        for (int d = k.d0 + threadIdx.x; d < k.d1; d += blockDim.x) {
            double t = D.t64[d];
            double u = D.precond == FG_PRECOND_DIAG ? t * D.invd64[d]
                     : precond_separate(D.precond) ? D.u64[d] : t;
            double bd = D.b[d];
            double r = -1.0 * (u + -1.0 * bd);
            D.r64[d] = r;
            a0 += r * r;
            if (has_f) {
                double s = D.ftrue[d] - t;
                a1 += s * s;
                if (first) a3 += D.ftrue[d] * D.ftrue[d];
            }
            if (first) a2 += bd * bd;
        }
        a0 = warp_sum(a0); a1 = warp_sum(a1); a2 = warp_sum(a2); a3 = warp_sum(a3);
        if (lane == 0) { red[0][warp] = a0; red[1][warp] = a1; red[2][warp] = a2; red[3][warp] = a3; }
        __syncthreads();
        if (threadIdx.x < 4) {
            double s = 0;
            for (int w = 0; w < kThreads / 32; ++w) s += red[threadIdx.x][w];
            D.part[k.part * kPartStride + threadIdx.x] = s;
        }
        if (last_part(D, 0)) {
            reduce_parts(D, 4, tot);
            if (threadIdx.x == 0) {
                SysState *st = D.st;
                double r0 = sqrt(tot[0]);
                if (st->first) {
                    st->normb = sqrt(tot[2]);
                    st->fnorm = sqrt(tot[3]);
                    st->eps = D.mixed ? D.tol : D.tol * st->normb;
                    st->first = 0;
                }
                double rel_true = has_f ? (st->fnorm > 0 ? sqrt(tot[1]) / st->fnorm : sqrt(tot[1])) : NAN;
                double rel_pre = st->normb > 0 ? r0 / st->normb : r0;
                st->true_res = rel_true;
                st->r0 = r0;
                st->steps = 0;
                bool stop = false;
                if (!(r0 > 0.0)) {                      // exact (or empty) right-hand side
                    stop = true;
                    st->converged = (r0 == 0.0);
                    if (!(r0 == 0.0)) st->status = FG_ERR_BREAKDOWN;
                    st->rho = r0;
                } else if (D.mixed) {
                    double m = has_f ? rel_true : rel_pre;
                    if (m <= D.tol) { stop = true; st->converged = 1; }
                    else if (st->cycles >= D.lmax) { stop = true; st->status = FG_ERR_NOTCONV; }
                    st->target = D.inner_tol * r0;
                }
                if (stop) { st->live = 0; st->in_cycle = 0; }
                else {
                    st->in_cycle = 1;
                    D.g[0] = r0;                        // e[0] = ||r||
                    st->rho = r0;
                }
            }
        }
    }
}

// v0 = r * (1 / ||r||) (pgmres.c:78-81)
template <typename TV>
__device__ __forceinline__ TV to_basis(double v)
{
    if constexpr (std::is_same<TV, __half>::value) return __float2half_rn((float)v);
    else return (TV)v;
}

// v_0 = r / ||r||, stored as sigma v_0 (sigma = 1 unless the basis is FP16)
template <typename T, typename TV = T>
__global__ void __launch_bounds__(kThreads)
k_scale_v0(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch)
{
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->in_cycle) continue;
        const double sc = 1.0 / D.st->r0;
        TV *V0 = (TV *)D.V;
        if (k.part == 0 && threadIdx.x == 0) D.vscale[0] = D.vsci;
        for (int d = k.d0 + threadIdx.x; d < k.d1; d += blockDim.x) {
            const T v = (T)(sc * D.r64[d]);
            V0[d] = to_basis<TV>((double)D.vsc * (double)v);
        }
    }
}

#include "arnoldi.cuh"

// final true residual: t64 holds A x
__global__ void __launch_bounds__(kThreads)
k_final(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch)
{
    __shared__ double red[kThreads / 32];
    __shared__ double tot[1];
    const int total = *nch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        double a = 0;
        for (int d = k.d0 + threadIdx.x; d < k.d1; d += blockDim.x) {
            double t = D.t64[d];
            if (D.ftrue) { double s = D.ftrue[d] - t; a += s * s; }
        }
        a = warp_sum(a);
        if (lane == 0) red[warp] = a;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0;
            for (int w8 = 0; w8 < kThreads / 32; ++w8) s += red[w8];
            D.part[k.part * kPartStride] = s;
        }
        if (last_part(D, 5)) {
            reduce_parts(D, 1, tot);
            if (threadIdx.x == 0) {
                SysState *st = D.st;
                st->true_res = D.ftrue ? (st->fnorm > 0 ? sqrt(tot[0]) / st->fnorm : sqrt(tot[0])) : NAN;
            }
        }
    }
}

__global__ void k_init_state(const SysDev *__restrict__ sys, int nsys)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    SysState *st = sys[s].st;
    memset(st, 0, sizeof(SysState));
    st->live = 1;
    st->first = 1;
    st->status = FG_OK;
    for (int c = 0; c < 8; ++c) sys[s].counter[c] = 0u;
}

// live flags of all systems into one array (pinned host memory)
__global__ void k_live(const SysDev *__restrict__ sys, int nsys, int *out)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nsys) out[s] = sys[s].st->live;
}

// states of all systems into one array (pinned host memory)
__global__ void k_states(const SysDev *__restrict__ sys, int nsys, SysState *out)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nsys) out[s] = *sys[s].st;
}

// ---------------------------------------------------------------- host side
int sm_count()
{
    constexpr int kKnown = 64;
    static std::atomic<int> known[kKnown];
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < kKnown && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) return 1;
    if (dev >= 0 && dev < kKnown) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

namespace {

// the matvec kernel of an S x S launch: 3x3, the pair kernel, or per element
template <int S, typename TA, bool PAIRS>
static auto pick_mv()
{
    if constexpr (S == 3) return k_ebe_mv3<TA>;
    else if constexpr (PAIRS && mvb_rows<S, TA>() > 0) return k_ebe_mvb<S, TA>;
    else return k_ebe_mv<S, TA>;
}

struct MvLaunch {
    // Persistent CTAs: as many as fit on the GPU (their dynamic shared memory,
    // mv_smem_bytes, decides how many per SM), at most one per patch.
    template <typename TA>
    static void go(int S, int nitems, cudaStream_t st, const SysDev *sys, const EChunk *ch, const int *nch,
                   const double *x, double *y, int maxdof)
    {
        switch (S) {
        case 3: run<3, TA>(nitems, st, sys, ch, nch, x, y, maxdof); break;
        case 6: run<6, TA>(nitems, st, sys, ch, nch, x, y, maxdof); break;
        case 9: run<9, TA>(nitems, st, sys, ch, nch, x, y, maxdof); break;
        case 12: run<12, TA>(nitems, st, sys, ch, nch, x, y, maxdof); break;
        }
    }
    template <int S, typename TA>
    static void run(int nitems, cudaStream_t st, const SysDev *sys, const EChunk *ch, const int *nch, const double *x,
                    double *y, int maxdof)
    {
        const size_t smem = mv_smem_bytes(S, maxdof, sizeof(TA));
        // FP64 S x S blocks: a thread per (element, row) (the FP64 pipe wants
        // every warp slot); FP32: a thread per element (its x values
        // gathered once, not once per row)
        // the pair kernel only for colour launches of up to two waves of the
        // per-element kernel (3 CTAs per SM): FP64 12x12 Euler 513^2 (7
        // launches of ~290-512 patches) 2.02 -> 2.46 TB/s, but NS 1025^2
        // (~1170 a launch) 3.23 -> 2.83 TB/s; both give the same sums
        constexpr bool can_pair = S > 3 && mvb_rows<S, TA>() > 0;
        const bool pairs = can_pair && nitems <= 6 * sm_count();
        auto kern = pairs ? pick_mv<S, TA, true>() : pick_mv<S, TA, false>();
        const int nt = pairs ? kMvbThreads : kThreads;
        // the attribute and the occupancy are cached per kernel (last
        // shared-memory size seen); they are host-side queries only
        static std::mutex mu;
        static size_t set_bytes[2] = {0, 0}, occ_bytes[2] = {0, 0};
        static int occ_cached[2] = {1, 1};
        const int w = pairs ? 1 : 0;
        int occ;
        {
            std::lock_guard<std::mutex> lk(mu);
            if (smem > set_bytes[w]) {
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                set_bytes[w] = smem;
            }
            if (smem != occ_bytes[w]) {
                int o = 0;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, nt, smem);
                occ_cached[w] = std::max(o, 1);
                occ_bytes[w] = smem;
            }
            occ = occ_cached[w];
        }
        const int g = std::max(1, std::min(nitems, occ * sm_count()));
        kern<<<g, nt, smem, st>>>(sys, ch, nch, x, y, maxdof);
    }
};

void launch_blockdiag(int B, dim3 g, cudaStream_t st, const SysDev *sys, const NChunk *ch, const int *nch)
{
    switch (B) {
    case 2: k_blockdiag<2><<<g, kThreads, 0, st>>>(sys, ch, nch); break;
    case 3: k_blockdiag<3><<<g, kThreads, 0, st>>>(sys, ch, nch); break;
    case 4: k_blockdiag<4><<<g, kThreads, 0, st>>>(sys, ch, nch); break;
    }
}

// a CTA a chunk: the hardware hands them out as CTAs finish
inline dim3 grid_for(int nchunks) { return dim3((unsigned)std::max(1, nchunks)); }

// Batches below this: what a member's sums depend on follows its own size only
// (parts of kPartMin, part_dofs_for).
constexpr long long kSoloDofs = 32768;

int parts_for(int n, int part_dofs = kPartMax)
{
    int p = (n + part_dofs - 1) / part_dofs;
    return std::max(1, std::min(kMaxParts, p));
}

}  // namespace

// ---------------------------------------------------------------- autotuner
// Measured launch shapes of a batch's streaming cycles, chosen by fg_autotune and cached per
// (block size, precision, batch-size class = floor(log2(batch dofs))) for
// the process: the dof-part size of the Krylov kernels and, for 3x3
// blocks in FP32, the matvec's work items (four rows a thread or one).  A batch
// with no cached choice, or one that runs on chip, uses the built-in rule.
struct TuneKey {
    int S, mixed, vhalf, cls;
    bool operator<(const TuneKey &o) const
    {
        return std::tie(S, mixed, vhalf, cls) < std::tie(o.S, o.mixed, o.vhalf, o.cls);
    }
};
static std::mutex g_tune_mu;
static std::map<TuneKey, fg_tune_choice> g_tune;
// set by the autotuner while it times a candidate (this thread only)
static thread_local const fg_tune_choice *t_tune_force = nullptr;

static long long batch_dofs(const std::vector<BatchMember> &mem)
{
    long long tot = 0;
    for (auto &m : mem) tot += m.s->topo.n;
    return tot;
}
static TuneKey tune_key(int S, const SolveConfig &cfg, long long dofs)
{
    int cls = 0;
    while ((2LL << cls) <= std::max(1LL, dofs)) ++cls;
    return {S, cfg.mixed, cfg.vhalf, cls};
}
// the tuned choice of a batch, or nullptr
static bool tuned_choice(const std::vector<BatchMember> &mem, const SolveConfig &cfg, fg_tune_choice &out)
{
    if (t_tune_force) { out = *t_tune_force; return true; }
    if (mem.empty()) return false;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find(tune_key(mem[0].s->topo.S, cfg, batch_dofs(mem)));
    if (it == g_tune.end()) return false;
    out = it->second;
    return true;
}

namespace {

// part size of a batch (multiple of 8 dofs): the tuned one, else kPartMin below
// kSoloDofs, 2 sqrt(batch dofs) up to 64k dofs and 4 sqrt above (where a part's sums are
// split among CTAs), rounded to the nearest power of two, within [kPartMin,
// kPartMax].  A batch that gives
// every resident CTA (3 an SM; FP64, which splits the sums, 4) a part of 1024 dofs
// (a pass of its threads) takes the smallest multiple of that with which the
// parts fill whole rounds of CTAs: 4.0 M dofs FP32 on 152 SMs, a step with 8192
// dofs in 506 parts 173 us, with 9216 in 452 parts 156; 3 M FP64 391 -> 362.
int part_dofs_for(const std::vector<BatchMember> &mem, const SolveConfig &cfg, bool tuned)
{
    fg_tune_choice tc;
    if (tuned && tuned_choice(mem, cfg, tc) && tc.part_dofs > 0) return tc.part_dofs & ~7;
    const long long dofs = std::max(1LL, batch_dofs(mem)), round = (cfg.mixed ? 3LL : 4LL) * sm_count();
    if (dofs > 1024 * round) {
        for (long long rounds = 1;; ++rounds)
            for (int pd = 1024; pd <= kPartMax; pd += 1024) {
                if (dofs > rounds * round * pd) continue;
                long long parts = 0;
                for (auto &m : mem) parts += parts_for(m.s->topo.n, pd);
                if (parts <= rounds * round) return pd;
            }
    }
    if (dofs < kSoloDofs) return kPartMin;
    const double tot = (double)dofs;
    const long long pd = 1LL << (int)std::lround(std::log2((tot > 65536.0 ? 4.0 : 2.0) * std::sqrt(tot)));
    return (int)std::max<long long>(kPartMin, std::min<long long>(kPartMax, pd));
}

// Units per work item of the matvec: one row per thread (256 / ndof units)
// while that leaves a wave of CTAs or less, so that small systems spread out,
// else four rows per thread.  A tuned choice can pin either (mv3_pipeline 0:
// always one row per thread); the sums are the same.
int unit_chunk(const std::vector<BatchMember> &mem, const SolveConfig &cfg, bool tuned)
{
    fg_tune_choice tc;
    const int B = mem[0].s->topo.ndof, one = 32 / B * (kThreads / 32);
    if (tuned && tuned_choice(mem, cfg, tc) && tc.mv3_pipeline == 0) return one;
    return batch_dofs(mem) > 8LL * kThreads * sm_count() ? 4 * one : one;
}

}  // namespace

// Chunk tables of one batch (device copies + host counts).
struct Plan {
    int nsys = 0, S = 3, B = 1;
    int precond = FG_PRECOND_NONE, ilu_g = 4;
    int n_dch = 0, n_nch = 0, n_ilu = 0, n_ilub = 0, n_spb = 0, n_spi = 0;
    // device tables, all in one block of the run's arena
    struct Span {
        void *p = nullptr;
        template <class T> T *as() const { return static_cast<T *>(p); }
    };
    Span sysdev, dchunks, dcount, nchunks, ncount;
    Span cyc_items;                                // on-chip cycle: (system, rank) of its CTAs
    std::vector<CycBin> bins;                      // its launches (none: the cycle streams)
    bool solo = false;                             // fewer than kSoloDofs equations
    bool rprec = false;                            // a right preconditioner (SGSe) before every matvec
    Span ilu_fwd, ilu_bwd, ilu_ctr;                // sync-free ILU(0) substitutions
    Span ilu_ws;                                 // block-Jacobi: (system, block) items, a warp each
    int n_ilw = 0, ilu_wx = 0, ilu_we = 0;         // items, rows of the largest block (0: level-scheduled
                                                   // path), entries of the longest chunk
    Span sp_blocks, sp_ifaces;                   // SPIKE (system, block) and (system, interface) items
};

static int choose_engine(const std::vector<BatchMember> &mem, const SolveConfig &cfg, std::vector<SysDev> &hs,
                         const std::vector<int> &live, int B, cudaStream_t st);
static size_t items_room(const std::vector<BatchMember> &mem, const SolveConfig &cfg, int B);

// cycles: restart cycles will run (else only residuals)
static int build_plan(Plan &P, std::vector<BatchMember> &mem, const SolveConfig &cfg, std::vector<SysDev> &hs,
                      bool cycles, PlanArena &arena, cudaStream_t st)
{
    int r;
    P.nsys = (int)mem.size();
    P.S = mem[0].s->topo.S;
    P.B = mem[0].s->topo.ndof;
    for (auto &m : mem)
        if (m.s->topo.S != P.S) { set_error("a batch must hold systems of one block size"); return FG_ERR_ARG; }
    std::vector<DChunk> dch;
    std::vector<NChunk> nch;
    P.rprec = cfg.precond == FG_PRECOND_SGSE;
    P.solo = batch_dofs(mem) < kSoloDofs;
    if (cycles && (r = choose_engine(mem, cfg, hs, {}, P.B, st))) return r;
    // (a tuned choice is one for the streaming kernels)
    bool chip = false;
    for (const SysDev &D : hs) chip = chip || D.cy_g > 0;
    const int pdofs = part_dofs_for(mem, cfg, !chip);
    const int uchunk = unit_chunk(mem, cfg, !chip);
    for (int s = 0; s < P.nsys; ++s) {
        int n = mem[s].s->topo.n;
        hs[s].nparts = parts_for(n, pdofs);
        int np = hs[s].nparts;
        // part boundaries on multiples of 8 dofs (16-byte packs in FP16, FP32 and FP64)
        for (int p = 0; p < np; ++p) {
            int d0 = (int)((long long)n * p / np) & ~7;
            int d1 = p + 1 == np ? n : (int)((long long)n * (p + 1) / np) & ~7;
            dch.push_back({s, p, d0, d1});
        }
        const int nn = mem[s].s->topo.nunits;
        for (int a = 0; a < nn; a += uchunk) nch.push_back({s, a, std::min(a + uchunk, nn)});
    }
    std::vector<CycItem> cyc;
    if (cycles) gang_items(hs, {}, P.B, !cfg.mixed, cyc, P.bins);
    P.n_dch = (int)dch.size();
    P.n_nch = (int)nch.size();
    P.precond = cfg.precond;
    for (auto &m : mem)
        if (m.s->op != mem[0].s->op) { set_error("a batch must use one operator kind"); return FG_ERR_ARG; }
    // ILU(0) substitutions: one item per pass of a system's level order
    // (forward and backward lists), systems interleaved
    std::vector<int2> fwd, bwd, wit;
    if (cfg.precond == FG_PRECOND_ILU0) {
        int maxp = 0;
        for (int s = 0; s < P.nsys; ++s) {
            maxp = std::max({maxp, mem[s].s->ilu_nfpass, mem[s].s->ilu_nbpass});
            P.ilu_g = std::max(P.ilu_g, mem[s].s->ilu_g);
        }
        for (int q = 0; q < maxp; ++q)
            for (int s = 0; s < P.nsys; ++s) {
                if (q < mem[s].s->ilu_nfpass) fwd.push_back(make_int2(s, q));
                if (q < mem[s].s->ilu_nbpass) bwd.push_back(make_int2(s, q));
            }
        P.n_ilu = (int)fwd.size();
        P.n_ilub = (int)bwd.size();
        // every member block-Jacobi with blocks small enough: a warp per block
        int wx = 0, we = 1;
        bool ws = true;
        for (int s = 0; s < P.nsys && ws; ++s) {
            const int rows = ilu_ws_rows(mem[s].s);
            ws = rows > 0;
            wx = std::max(wx, rows);
            we = std::max(we, mem[s].s->ilu_maxrow);
        }
        we *= kIluWsChunk;
        if (ws && P.nsys > 0) {
            for (int s = 0; s < P.nsys; ++s) {
                const int np = std::max(1, std::min(mem[s].s->ilu_blocks, mem[s].s->topo.n));
                for (int q = 0; q < np; ++q) wit.push_back(make_int2(s, q));
            }
            P.n_ilw = (int)wit.size();
            P.ilu_wx = wx;
            P.ilu_we = we;
        }
    }
    // SPIKE: one CTA per block and per interface of every member
    std::vector<int2> spb, spi;
    if (cfg.precond == FG_PRECOND_SPIKE)
        for (int s = 0; s < P.nsys; ++s) {
            const int np = mem[s].s->sp_P;
            for (int q = 0; q < np; ++q) spb.push_back(make_int2(s, q));
            for (int q = 0; q + 1 < np; ++q) spi.push_back(make_int2(s, q));
        }
    P.n_spb = (int)spb.size();
    P.n_spi = (int)spi.size();
    // one block, one copy: the tables in pinned staging, in order
    struct Piece { Plan::Span *to; const void *from; size_t bytes, room; };
    const int zeros[16] = {0};
    auto piece = [](Plan::Span &to, const auto &v, size_t least = 0) {
        const size_t e = sizeof(v[0]);
        return Piece{&to, v.data(), e * v.size(), e * std::max(v.size(), least)};
    };
    const Piece all[] = {
        piece(P.sysdev, hs), piece(P.dchunks, dch), {&P.dcount, &P.n_dch, sizeof(int), sizeof(int)},
        piece(P.nchunks, nch), {&P.ncount, &P.n_nch, sizeof(int), sizeof(int)},
        piece(P.cyc_items, cyc, cycles ? items_room(mem, cfg, P.B) : 0), piece(P.ilu_fwd, fwd), piece(P.ilu_bwd, bwd),
        {&P.ilu_ctr, zeros, sizeof(zeros), sizeof(zeros)}, piece(P.ilu_ws, wit), piece(P.sp_blocks, spb),
        piece(P.sp_ifaces, spi)};
    size_t bytes = 0;
    for (const Piece &q : all) bytes += (q.room + 255) & ~(size_t)255;
    if ((r = arena.ensure(bytes, P.nsys))) return r;
    size_t at = 0;
    for (const Piece &q : all) {
        q.to->p = arena.dev.as<unsigned char>() + at;
        if (q.bytes) std::memcpy(arena.host + at, q.from, q.bytes);
        at += (q.room + 255) & ~(size_t)255;
    }
    FG_CUDA(cudaMemcpyAsync(arena.dev.p, arena.host, at, cudaMemcpyHostToDevice, st));
    return FG_OK;
}

// Room for `bytes` of tables and the flags and states of n members.  The
// staging is rewritten only between cycles: a copy of it that may still be in
// flight then (tables of a batch that changed twice) is followed by one of the
// new tables before any kernel reads them.
int PlanArena::ensure(size_t bytes, int n)
{
    int r;
    if (dev.bytes < bytes || host_bytes < bytes || members < n) {
        bytes = std::max(bytes + bytes / 2, (size_t)16384);
        n = std::max(n, 8);
        if ((r = dev.alloc(bytes))) return r;
        if (host) cudaFreeHost(host);
        host = nullptr;
        host_bytes = 0;                    // (should the next line fail, the next run asks again)
        members = 0;
        const size_t tail = 2 * sizeof(int) * (size_t)n + sizeof(SysState) * (size_t)n + 64;
        FG_CUDA(cudaMallocHost(&host, bytes + tail));
        host_bytes = bytes;
        members = n;
        states = reinterpret_cast<SysState *>(host + (bytes + 15) / 16 * 16);
        live = reinterpret_cast<int *>(states + n);
    }
    return FG_OK;
}
PlanArena::~PlanArena()
{
    if (host) cudaFreeHost(host);
}

// Enqueue the matvec: mode 0 (x -> t64, FP64, gate live), mode 1 (V[step]
// -> w = M^-1 A v, T, gate in_cycle; a preconditioner with kernels of its own
// gets t = A v instead), mode 2 (V[0] -> t, T, every member), mode 3
// (x -> t64, FP64, every member).  Returns the number of kernels.
// TV: storage type of the basis vector read in mode 1 (the Arnoldi step)
template <typename T, typename TV = T>
static int enqueue_matvec(const Plan &P, int mode, int step, cudaStream_t st)
{
    const bool f64 = mode == 0 || mode == 3;
    const int gate = mode == 0 ? 0 : mode == 1 ? 1 : -1;
    const bool own = P.precond == FG_PRECOND_ILU0 || P.precond == FG_PRECOND_SPIKE || P.precond == FG_PRECOND_LUE ||
                     P.precond == FG_PRECOND_SGSE;
    // pgmres.c:61,93: v = precondR(x or u_i) before the matvec (SGSe), into r64
    int in = f64 ? 0 : 1, kr = 0;
    if (P.rprec && (mode == 0 || mode == 1)) {
        launch_elem_prec(P.sysdev.as<SysDev>(), P.nsys, 3, mode == 0 ? 0 : 1, step, st);
        in = 3;
        kr = 1;
    }
    const int prec = f64 || sizeof(T) == 8 ? 64 : sizeof(TV) == 2 ? 16 : 32;
    const int out = f64 ? 0 : mode == 1 && !own ? 2 : 1;
    return kr + launch_rows_mv(P.B, prec, P.sysdev.as<SysDev>(), P.nchunks.as<NChunk>(), P.ncount.as<int>(), P.n_nch,
                               gate, in, out, step, st);
}

// M^-1 applied after a matvec: sel 0 (t64 -> u64, FP64) or 1 (t -> w, T).
template <typename T>
static int enqueue_precond(const Plan &P, int sel, cudaStream_t st)
{
    const SysDev *sys = P.sysdev.as<SysDev>();
    if (P.precond == FG_PRECOND_BLOCKDIAG) {
        if (sel == 1) return 0;                       // in the matvec
        launch_blockdiag(P.B, grid_for(P.n_nch), st, sys, P.nchunks.as<NChunk>(), P.ncount.as<int>());
        return 1;
    }
    if (P.precond == FG_PRECOND_LUE || P.precond == FG_PRECOND_SGSE) {   // FP64 only
        launch_elem_prec(sys, P.nsys, P.precond == FG_PRECOND_LUE ? 1 : 2, sel, 0, st);
        return 1;
    }
    if (P.precond == FG_PRECOND_ILU0 && P.n_ilw > 0) {
        const int fp32 = sel == 1 && sizeof(T) == 4;
        launch_ilu_ws(sys, P.ilu_ws.as<int2>(), P.n_ilw, sel, 0, fp32, P.ilu_g, P.ilu_wx, P.ilu_we, st);
        launch_ilu_ws(sys, P.ilu_ws.as<int2>(), P.n_ilw, sel, 1, fp32, P.ilu_g, P.ilu_wx, P.ilu_we, st);
        return 2;
    }
    if (P.precond == FG_PRECOND_ILU0) {
        int *ctr = P.ilu_ctr.as<int>(), *err = ctr + 4;
        const int fp32 = sel == 1 && sizeof(T) == 4;
        launch_ilu_pending(sys, P.dchunks.as<DChunk>(), P.dcount.as<int>(), P.n_dch, sel, fp32, st);
        launch_ilu_solve(sys, P.ilu_fwd.as<int2>(), P.n_ilu, ctr, err, sel, 0, fp32, P.ilu_g, st);
        launch_ilu_solve(sys, P.ilu_bwd.as<int2>(), P.n_ilub, ctr, err, sel, 1, fp32, P.ilu_g, st);
        return 3;
    }
    if (P.precond == FG_PRECOND_SPIKE) {
        const int fp32 = sel == 1 && sizeof(T) == 4;
        launch_spike_apply(sys, P.sp_blocks.as<int2>(), P.n_spb, P.sp_ifaces.as<int2>(), P.n_spi, sel, fp32, st);
        return P.n_spi > 0 ? 3 : 1;
    }
    return 0;
}

// One restart cycle for every member; returns the number of kernels.  TV
// is the basis' storage type (T, or FP16 under FP32 arithmetic).  A batch
// whose bases fit the chip runs its Arnoldi steps in a kernel, or a few
// (cycle.cu, choose_engine), any other streams through the pass kernels below.
template <typename T, typename TV = T>
static int enqueue_cycle(const Plan &P, const SolveConfig &cfg, int *live, cudaStream_t st)
{
    const SysDev *sys = P.sysdev.as<SysDev>();
    const DChunk *dc = P.dchunks.as<DChunk>();
    const int *nd = P.dcount.as<int>();
    int k = enqueue_matvec<T>(P, 0, 0, st);
    k += enqueue_precond<T>(P, 0, st);
    k_start<<<grid_for(P.n_dch), kThreads, 0, st>>>(sys, dc, nd);
    ++k;
    for (const CycBin &b : P.bins)
        k += launch_cycle(P.B, sizeof(T) == 8, b.spill, sys, P.cyc_items.as<CycItem>() + b.first, b.ctas, b.smem, st);
    if (P.bins.empty()) {
        const dim3 gd = grid_for(P.n_dch);
        // Few parts: several CTAs each, up to eight CTAs an SM in all.  FP32: none
        // once parts fill two CTAs an SM (4.0 M dofs in 452 parts, CTAs a part in
        // the two passes 1 and 1: 156 us a step, 2 and 2: 163, 4 and 4: 174); FP64 is bound by
        // its pipe and wants it evenly loaded (3 M dofs in 600 parts, 1 and 1: 397,
        // 2 and 2: 373, 4 and 2: 362).
        const int fill = 8 * sm_count() / std::max(1, P.n_dch), ways = std::min(16, fill * (sizeof(T) == 8 ? 2 : 1));
        const bool split = sizeof(T) == 8 || P.n_dch < 2 * sm_count();
        // (a part's norm depends on the CTAs it is split among in pass 2, not on those of pass 1)
        const int yd = split ? std::max(1, ways) : 1;
        const int yo = P.solo ? kMaxSplit : split ? std::max(1, std::min(kMaxSplit, fill)) : 1;
        k_scale_v0<T, TV><<<gd, kThreads, 0, st>>>(sys, dc, nd);
        ++k;
        for (int i = 0; i < cfg.kmax - 1; ++i) {
            k += enqueue_matvec<T, TV>(P, 1, i, st);
            k += enqueue_precond<T>(P, 1, st);
            k_dots<T, TV><<<dim3(gd.x, std::min(yd, (i + 4) / 4)), kThreads, 0, st>>>(sys, dc, nd, i);
            k_orth<T, TV><<<dim3(gd.x, yo), kThreads, 0, st>>>(sys, dc, nd, i);
            k += 2;
            if constexpr (!std::is_same<T, TV>::value) {
                k_normalize<T, TV><<<gd, kThreads, 0, st>>>(sys, dc, nd, i);
                ++k;
            }
        }
        k_update<T, TV><<<gd, kThreads, 0, st>>>(sys, dc, nd);
        ++k;
    }
    k_live<<<(P.nsys + 255) / 256, 256, 0, st>>>(sys, P.nsys, live);
    return k + 1;
}

// The gang of a member's on-chip restart cycle (0: it streams): the
// preconditioner must act on one node, the basis must be kept in the
// arithmetic's type and fit.
static bool chip_config(const SolveConfig &cfg)
{
    return !cfg.vhalf && (cfg.precond == FG_PRECOND_NONE || cfg.precond == FG_PRECOND_DIAG ||
                          cfg.precond == FG_PRECOND_BLOCKDIAG);
}
static int member_gang(const fg_system *s, const SolveConfig &cfg, bool dense)
{
    return chip_config(cfg) ? gang_size(s, cfg.kmax, !cfg.mixed, dense) : 0;
}

// CTAs that the members' on-chip launches may hold at most, now or as members stop
static size_t items_room(const std::vector<BatchMember> &mem, const SolveConfig &cfg, int B)
{
    const size_t room = gang_ctas(B, !cfg.mixed);
    size_t sum = 0;
    for (const BatchMember &m : mem) {
        const int g = member_gang(m.s, cfg, true);
        sum += g ? std::max(g, member_gang(m.s, cfg, false)) : room;
    }
    return chip_config(cfg) ? std::max(room, sum) : 0;
}

// The basis in global memory: kmax vectors, which the streaming kernels
// use, or those that a gang of the whole chip keeps outside (more where
// prescribed dofs count among the units).
static size_t basis_bytes(const fg_system *s, int kmax, int mode)
{
    const size_t w = mode == 0 ? 8 : mode == 2 ? 2 : 4, all = w * (size_t)s->n_pad * kmax;
    const int js = mode == 2 ? 0 : gang_spill(s, kmax, mode == 0);
    return std::max(all, gang_spill_bytes(s, kmax, gang_ctas(s->topo.ndof, mode == 0, true), js, mode == 0));
}

// mode: 0 FP64, 1 FP32 basis, 2 FP16 basis (mixed precision in both).  All
// that a cycle may need is allocated before the first one, wherever it runs,
// but the exchange blocks of the gangs (choose_engine).
static int ensure_workspace(fg_system *s, int kmax, int mode)
{
    Workspace &w = s->ws;
    if (w.kmax >= kmax && w.mixed == mode) return FG_OK;
    w.kmax = 0;
    w.mixed = -1;
    w.v_lent = false;
    size_t np = (size_t)s->n_pad, ts = mode ? sizeof(float) : sizeof(double);
    int r;
    if ((r = w.V.alloc(basis_bytes(s, kmax, mode))) || (r = w.w.alloc(ts * np)) || (r = w.t.alloc(ts * np)) ||
        (r = w.x.alloc(8 * np)) || (r = w.b.alloc(8 * np)) || (r = w.ftrue.alloc(8 * np)) ||
        (r = w.r64.alloc(8 * np)) || (r = w.t64.alloc(8 * np)) || (r = w.u64.alloc(8 * np)) ||
        (r = w.small.alloc(8 * ((size_t)(kmax + 1) * kmax + 7 * (kmax + 1) + (size_t)kmax * kmax))) ||
        (r = w.part.alloc(8 * (size_t)kMaxParts * kPartStride)) ||
        (r = w.counter.alloc(sizeof(unsigned) * 8)) || (r = w.state.alloc(sizeof(SysState))))
        return r;
    w.kmax = kmax;
    w.mixed = mode;
    return FG_OK;
}
static SysDev make_desc(fg_system *s, const SolveConfig &cfg, bool has_f)
{
    const Topology &t = s->topo;
    Workspace &w = s->ws;
    SysDev D{};
    D.n = t.n; D.n_pad = s->n_pad; D.nel = t.nel; D.nel_pad = s->nel_pad; D.S = t.S; D.ndof = t.ndof;
    D.ncol = t.ncol; D.nparts = parts_for(t.n); D.nnodes = t.nnodes;
    D.kmax = cfg.kmax; D.lmax = cfg.lmax; D.mixed = cfg.mixed; D.precond = cfg.precond;
    D.tol = cfg.tol; D.inner_tol = cfg.inner_tol;
    D.vhalf = cfg.vhalf;
    D.vsc = D.vsci = 1.0f;
    if (cfg.vhalf) {   // unit vectors times 2^floor(log2 sqrt n): entries of order 1 in FP16
        const int e = (int)std::floor(0.5 * std::log2((double)std::max(t.n, 1)));
        D.vsc = std::ldexp(1.0f, e);
        D.vsci = std::ldexp(1.0f, -e);
    }
    D.lm = s->lm.as<int>(); D.A64 = s->A64.as<double>(); D.A32 = s->A32.as<float>();
    set_patch_fields(D, s);
    D.invd64 = s->invd64.as<double>(); D.invd32 = s->invd32.as<float>();
    D.node_dof = s->node_dof.as<int>(); D.ibd64 = s->ibd64.as<double>(); D.ibd32 = s->ibd32.as<float>();
    D.x = w.x.as<double>(); D.b = w.b.as<double>(); D.ftrue = has_f ? w.ftrue.as<double>() : nullptr;
    D.r64 = w.r64.as<double>(); D.t64 = w.t64.as<double>(); D.u64 = w.u64.as<double>();
    D.V = w.V.p; D.w = w.w.p; D.t = w.t.p;
    double *sm = w.small.as<double>();
    D.H = sm;
    D.g = sm + (size_t)(cfg.kmax + 1) * cfg.kmax;
    D.cs = D.g + (cfg.kmax + 1);
    D.sn = D.cs + (cfg.kmax + 1);
    D.hbuf = D.sn + (cfg.kmax + 1);
    D.y = D.hbuf + (cfg.kmax + 1);
    D.hcol = D.y + (cfg.kmax + 1);
    D.vscale = D.hcol + (cfg.kmax + 1);
    D.G = D.vscale + (cfg.kmax + 1);
    D.part = w.part.as<double>();
    D.counter = w.counter.as<unsigned>();
    D.st = w.state.as<SysState>();
    return D;
}

int validate_member(fg_system *s, const SolveConfig &cfg)
{
    if (cfg.kmax < 2 || cfg.kmax > kMaxRestart) { set_error("kmax must be in [2, 60]"); return FG_ERR_ARG; }
    if (cfg.lmax < 1) { set_error("lmax must be >= 1"); return FG_ERR_ARG; }
    if (!s->blocks_ok) { set_error("solve before element blocks were set"); return FG_ERR_STATE; }
    if (cfg.precond != FG_PRECOND_NONE && s->precond != cfg.precond) {
        set_error("solve with a preconditioner that was not set up"); return FG_ERR_STATE;
    }
    if (cfg.precond == FG_PRECOND_BLOCKDIAG && s->topo.ndof < 2) {
        set_error("block-diagonal preconditioner needs ndof >= 2"); return FG_ERR_UNSUPPORTED;
    }
    if (s->op == FG_OP_CSR && !s->csr_ok) { set_error("CSR operator selected but not set up"); return FG_ERR_STATE; }
    if (cfg.precond == FG_PRECOND_ILU0 && s->op != FG_OP_CSR) {
        set_error("ILU(0) needs the CSR operator (fg_set_operator(FG_OP_CSR))"); return FG_ERR_STATE;
    }
    if ((cfg.precond == FG_PRECOND_LUE || cfg.precond == FG_PRECOND_SGSE) &&
        (cfg.mixed || s->topo.S != 3 || s->op != FG_OP_EBE)) {
        set_error("the element preconditioners LUe / SGSe run in FP64 on 3x3 EBE systems");
        return FG_ERR_UNSUPPORTED;
    }
    if (cfg.precond == FG_PRECOND_SPIKE && (s->op != FG_OP_CSR || !s->sp_ready)) {
        set_error("SPIKE needs the CSR operator and its set-up (fg_precond_setup)"); return FG_ERR_STATE;
    }
    return FG_OK;
}

size_t workspace_bytes(const fg_system *s, int kmax, int mixed)
{
    size_t np = (size_t)s->n_pad, ts = mixed ? 4 : 8;
    return ts * np * (kmax + 2) + 8 * np * 6 +
           8 * ((size_t)(kmax + 1) * kmax + 7 * (kmax + 1) + (size_t)kmax * kmax) +
           8 * (size_t)kMaxParts * kPartStride + 256 +
           gang_bytes(s, kmax, gang_ctas(s->topo.ndof, !mixed), !mixed);
}

int autotune(std::vector<fg_system *> &sys, const SolveConfig &cfg0, bool remeasure, bool lookup_only,
             fg_tune_choice *out)
{
    if (sys.empty()) { set_error("fg_autotune: empty batch"); return FG_ERR_ARG; }
    std::vector<BatchMember> mem;
    for (fg_system *s : sys) {
        if (!s) { set_error("fg_autotune: NULL system"); return FG_ERR_ARG; }
        if (s->topo.S != sys[0]->topo.S) { set_error("fg_autotune: a batch must hold one block size"); return FG_ERR_ARG; }
        if (!s->rhs_ok) { set_error("fg_autotune: system without a resident right-hand side"); return FG_ERR_STATE; }
        mem.push_back({s, s->rhs_b.as<double>(), s->rhs_f.as<double>(), nullptr});
    }
    SolveConfig cfg = cfg0;
    cfg.device_io = 1;
    cfg.use_graph = 0;
    cfg.precond = sys[0]->precond;
    const TuneKey key = tune_key(sys[0]->topo.S, cfg, batch_dofs(mem));
    if (!remeasure || lookup_only) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune.find(key);
        if (it != g_tune.end()) {
            *out = it->second;
            out->from_cache = 1;
            return FG_OK;
        }
        if (lookup_only) { set_error("fg_tune_lookup: no cached choice for this batch"); return FG_ERR_STATE; }
    }
    cudaStream_t st = sys[0]->stream;
    for (fg_system *s : sys) FG_CUDA(cudaStreamSynchronize(s->stream));
    std::vector<fg_tune_choice> cand;
    const int pds[] = {256, 512, 1024, 2048, 4096, 8192, 12288, 16384};
    const bool mv3_alt = sys[0]->topo.S == 3 && cfg.mixed && !cfg.vhalf;
    for (int pd : pds)
        for (int mv = 1; mv >= (mv3_alt ? 0 : 1); --mv) cand.push_back({pd, mv, 0.0, 0, 0});
    const char *tlog = getenv("FEMGPU_TUNE_LOG");
    const bool log = tlog && *tlog && *tlog != '0';
    cudaEvent_t e0, e1;
    FG_CUDA(cudaEventCreate(&e0));
    FG_CUDA(cudaEventCreate(&e1));
    fg_tune_choice best{};
    best.ms_per_cycle = 1e300;
    int r = FG_OK;
    std::vector<int> live;
    for (auto &c : cand) {
        t_tune_force = &c;
        {
            BatchRun run(cfg, st);
            for (auto &m : mem)
                if ((r = run.stage(m))) break;
            if (!r) r = run.commit();
            if (!r) r = run.cycle(false, live);                     // warm-up (first launches)
            if (!r) {
                cudaEventRecord(e0, st);
                r = run.cycle(false, live);
                cudaEventRecord(e1, st);
            }
            if (!r) {
                float ms = 0.f;
                cudaError_t ce = cudaEventSynchronize(e1);
                if (ce == cudaSuccess) ce = cudaEventElapsedTime(&ms, e0, e1);
                if (ce != cudaSuccess) r = cuda_fail(ce, "fg_autotune timing");
                c.ms_per_cycle = ms;
            }
        }
        t_tune_force = nullptr;
        if (r) break;
        if (log)
            fprintf(stderr, "fg_autotune: S=%d mixed=%d part_dofs=%d mv3_pipeline=%d: %.3f ms/cycle\n",
                    sys[0]->topo.S, cfg.mixed, c.part_dofs, c.mv3_pipeline, c.ms_per_cycle);
        if (c.ms_per_cycle < best.ms_per_cycle) best = c;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (r) return r;
    best.candidates = (int)cand.size();
    best.from_cache = 0;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune[key] = best;
    }
    *out = best;
    return FG_OK;
}

int tune_set(std::vector<fg_system *> &sys, const SolveConfig &cfg0, const fg_tune_choice &c)
{
    if (sys.empty()) { set_error("fg_tune_set: empty batch"); return FG_ERR_ARG; }
    std::vector<BatchMember> mem;
    for (fg_system *s : sys) {
        if (!s) { set_error("fg_tune_set: NULL system"); return FG_ERR_ARG; }
        if (s->topo.S != sys[0]->topo.S) { set_error("fg_tune_set: a batch must hold one block size"); return FG_ERR_ARG; }
        mem.push_back({s, nullptr, nullptr, nullptr});
    }
    if (c.part_dofs < kPartMin || c.part_dofs > kPartMax || c.part_dofs % 8 || (c.mv3_pipeline & ~1)) {
        set_error("fg_tune_set: part_dofs must be a multiple of 8 in [256, 16384], mv3_pipeline 0 or 1");
        return FG_ERR_ARG;
    }
    SolveConfig cfg = cfg0;
    cfg.precond = sys[0]->precond;
    fg_tune_choice k = c;
    k.from_cache = 0;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[tune_key(sys[0]->topo.S, cfg, batch_dofs(mem))] = k;
    return FG_OK;
}

void tune_clear()
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune.clear();
}

size_t request_bytes(const fg_system *s, int kmax, int mixed, bool time_loop)
{
    const Workspace &w = s->ws;
    const DevMem *held[] = {&w.V, &w.w, &w.t, &w.x, &w.b, &w.ftrue, &w.r64, &w.t64, &w.u64, &w.small, &w.part,
                            &w.counter, &w.state, &w.gang};
    size_t have = 0;
    for (auto *m : held) have += m->bytes;
    size_t b = s->bytes() - std::min(have, s->bytes()) + workspace_bytes(s, kmax, mixed) + rows_bytes(s, mixed != 0);
    if (time_loop) {
        const DevMem *loop[] = {&s->rhs_f, &s->rhs_b, &s->state_u, &s->state_a, &s->state_old};
        for (auto *m : loop)
            if (!m->p) b += 8 * (size_t)s->n_pad;
    }
    return b;
}

BatchRun::BatchRun(const SolveConfig &c, cudaStream_t s, PlanArena *a) : cfg(c), st(s), arena(a ? a : &own) {}

BatchRun::~BatchRun()
{
    if (exec) cudaGraphExecDestroy(exec);
    for (cudaEvent_t e : done)
        if (e) cudaEventDestroy(e);
}

// Workspace, cleared vectors and right-hand side of a new member (queued on
// the batch stream); the member joins at the next commit().
int BatchRun::stage(const BatchMember &m)
{
    fg_system *s = m.s;
    int r = validate_member(s, cfg);
    if (r) return r;
    if ((r = ensure_workspace(s, cfg.kmax, cfg.mixed + cfg.vhalf))) return r;
    if ((r = rows_refresh(s, cfg.mixed != 0, st))) return r;
    Workspace &w = s->ws;
    size_t vb = 8 * (size_t)s->n_pad;
    FG_CUDA(cudaMemsetAsync(w.x.p, 0, vb, st));
    if (w.gang.p) FG_CUDA(cudaMemsetAsync(w.gang.p, 0, w.gang.bytes, st));
    FG_CUDA(cudaMemsetAsync(w.small.p, 0, w.small.bytes, st));
    if (cfg.device_io) {
        FG_CUDA(cudaMemcpyAsync(w.b.p, m.B, 8 * (size_t)(s->topo.n + 1), cudaMemcpyDeviceToDevice, st));
        if (m.Ftrue) FG_CUDA(cudaMemcpyAsync(w.ftrue.p, m.Ftrue, 8 * (size_t)(s->topo.n + 1), cudaMemcpyDeviceToDevice, st));
    } else {
        // host vectors in reference numbering -> staging -> internal numbering
        size_t hb = 8 * (size_t)(s->topo.n + 1);
        FG_CUDA(cudaMemcpyAsync(w.r64.p, m.B, hb, cudaMemcpyHostToDevice, st));
        if ((r = permute_in(s, w.r64.as<double>(), w.b.as<double>(), st))) return r;
        if (m.Ftrue) {
            FG_CUDA(cudaMemcpyAsync(w.u64.p, m.Ftrue, hb, cudaMemcpyHostToDevice, st));
            if ((r = permute_in(s, w.u64.as<double>(), w.ftrue.as<double>(), st))) return r;
        }
    }
    mem.push_back(m);
    hs.push_back(make_desc(s, cfg, m.Ftrue != nullptr));
    ++pending;
    return FG_OK;
}

// Where the batch's restart cycles run, for the live members (all: empty).  On
// chip when gangs of the CTAs they like (gang_want) are resident together, or in a
// batch below kSoloDofs, in as many launches as these gangs take.
// Else as up to kMaxBins launches one behind the other, in which gangs are as
// small as their rows allow and a member that fits no chip has all of one with
// part of its basis outside.  Else streaming through global memory, all at once:
// a launch is about 9 us a step (FP64 20 to 50) whatever it holds up to 276k
// equations, while streaming takes 25 us (FP64 55) and little more for each
// further member.  Measured, streaming -> launches: 2 transport instances 53.9 ->
// 33.7 ms (FP64 100 -> 74), 4 65.9 -> 41.7, 10 in up to 3 launches 74.8 -> 71.5 (FP64
// 132 -> 126), in up to 4 74.9 (FP64 127), 16 119.5 -> 117.3, in up to 6 125.2.
constexpr int kMaxBins = 3;
// The choice for the live members (all: empty), written to hs where it
// changes.  Members with live given are in mid-solve: those on chip stay there (a
// gang's block has room for the largest gang that its system can get), those that
// stream move on chip if they now fit and their gangs' blocks can be had.
static int choose_engine(const std::vector<BatchMember> &mem, const SolveConfig &cfg, std::vector<SysDev> &hs,
                         const std::vector<int> &live, int B, cudaStream_t st)
{
    const int room = gang_ctas(B, !cfg.mixed), n = (int)mem.size();
    std::vector<int> g(n, 0), js(n, 0), bin(n, 0);
    std::vector<int> todo;
    for (int i = 0; i < n; ++i)
        if (live.empty() || live[i]) todo.push_back(i);
    // launches of the gangs, the largest first; a member that fits no chip has one of its own
    auto pack = [&] {
        std::stable_sort(todo.begin(), todo.end(), [&](int a, int b) { return g[a] > g[b]; });
        std::vector<int> left;
        for (int i : todo) {
            size_t b = 0;
            while (b < left.size() && (js[i] || left[b] < g[i])) ++b;
            if (b == left.size()) left.push_back(room);
            bin[i] = (int)b;
            left[b] = js[i] ? 0 : left[b] - g[i];
        }
        return (int)left.size();
    };
    const bool can = chip_config(cfg) && room > 0 && !t_tune_force;   // (the autotuner times streaming cycles)
    bool chip = can;
    long long sum = 0;
    const bool solo = batch_dofs(mem) < kSoloDofs;
    for (int i : todo)
        if (chip) {
            sum += g[i] = member_gang(mem[i].s, cfg, false);
            chip = g[i] > 0 && (solo || sum <= room);
        }
    if (chip) pack();
    else if (can) {
        chip = true;
        for (int i : todo) {
            g[i] = member_gang(mem[i].s, cfg, true);
            if (!g[i] && (js[i] = gang_spill(mem[i].s, cfg.kmax, !cfg.mixed)) > 0) g[i] = gang_ctas(B, !cfg.mixed, true);
            chip = chip && g[i] > 0;
        }
        chip = pack() <= kMaxBins && chip;
    }
    // no memory for the gangs: stream
    for (int i : todo) {
        if (!chip) break;
        Workspace &w = mem[i].s->ws;
        const int most = std::max(g[i], member_gang(mem[i].s, cfg, false));
        const size_t gb = gang_bytes(mem[i].s, cfg.kmax, most, !cfg.mixed);
        chip = (w.gang.bytes >= gb || w.gang.alloc(gb) == FG_OK) &&
               w.V.bytes >= gang_spill_bytes(mem[i].s, cfg.kmax, g[i], js[i], !cfg.mixed);
    }
    if (!chip) {
        cudaGetLastError();
        if (!live.empty()) return FG_OK;              // as they are
    }
    for (int i = 0; i < n; ++i) {
        fg_system *s = mem[i].s;
        Workspace &w = s->ws;
        // the streaming sweeps read packs across n and the sink at n: zeros, but
        // not where a gang kept its vectors
        if (!chip && w.v_lent) {
            FG_CUDA(cudaMemsetAsync(w.V.p, 0, w.V.bytes, st));
            w.v_lent = false;
        }
        hs[i].V = w.V.p;
        hs[i].cy_bin = bin[i];
        set_gang_fields(hs[i], s, cfg.kmax, chip ? g[i] : 0, chip ? js[i] : 0, !cfg.mixed);
        if (hs[i].cy_js > 0) w.v_lent = true;
    }
    return FG_OK;
}

// Rebuild the work tables for the current members and initialise the state
// of the members staged since the last commit.
int BatchRun::commit()
{
    if (exec) { cudaGraphExecDestroy(exec); exec = nullptr; }
    sched.clear();
    if (mem.empty()) { pending = 0; return FG_OK; }
    P = std::make_unique<Plan>();
    int r = build_plan(*P, mem, cfg, hs, true, *arena, st);
    if (r) return r;
    if (pending > 0) {
        int first = (int)mem.size() - pending;
        k_init_state<<<(pending + 127) / 128, 128, 0, st>>>(P->sysdev.as<SysDev>() + first, pending);
        FG_CUDA(cudaGetLastError());
        count_launches(1);
    }
    pending = 0;
    return FG_OK;
}

// One restart cycle of every member queued, its live flags to `flags`.
int BatchRun::enqueue(bool use_graph, int *flags)
{
    const Plan &Pl = *P;
    cudaError_t ce = cudaSuccess;
    auto queue = [&] {
        return cfg.vhalf ? enqueue_cycle<float, __half>(Pl, cfg, flags, st)
               : cfg.mixed ? enqueue_cycle<float>(Pl, cfg, flags, st) : enqueue_cycle<double>(Pl, cfg, flags, st);
    };
    if (!Pl.bins.empty()) use_graph = false;           // on chip: a few launches
    if (use_graph && !exec) {
        cudaGraph_t graph = nullptr;
        FG_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        graph_nodes = queue();
        ce = cudaStreamEndCapture(st, &graph);
        if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
        ce = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) { exec = nullptr; return cuda_fail(ce, "cudaGraphInstantiate"); }
    }
    if (use_graph) {
        ce = cudaGraphLaunch(exec, st);
        count_launches(graph_nodes);
    } else {
        count_launches(queue());
        ce = cudaGetLastError();
    }
    return ce == cudaSuccess ? FG_OK : cuda_fail(ce, "GMRES cycle");
}

// One restart cycle of every member; live[i] tells whether member i goes on.
int BatchRun::cycle(bool use_graph, std::vector<int> &live)
{
    live.assign(mem.size(), 0);
    if (mem.empty()) return FG_OK;
    int r = enqueue(use_graph, arena->live);
    if (r) return r;
    cudaError_t ce = cudaStreamSynchronize(st);
    if (ce != cudaSuccess) return cuda_fail(ce, "GMRES cycle");
    for (size_t i = 0; i < mem.size(); ++i) live[i] = arena->live[i];
    return reschedule(live);
}

// Restart cycles until every member stopped, at most `limit`.  A single
// system's next cycle is queued before its flag is read, so that the host's
// round trip does not show between cycles; the one queued last finds the
// system stopped and does nothing.
int BatchRun::run(bool use_graph, int limit)
{
    int r;
    if (mem.size() != 1 || use_graph_streams(use_graph)) {
        std::vector<int> live;
        for (int c = 0; c < limit; ++c) {
            if ((r = cycle(use_graph, live))) return r;
            int any = 0;
            for (int v : live) any |= v;
            if (!any) break;
        }
        return FG_OK;
    }
    for (cudaEvent_t &e : done)
        if (!e) FG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (int c = 0; c <= limit; ++c) {
        if (c < limit) {
            if ((r = enqueue(false, arena->live + (c & 1)))) return r;
            FG_CUDA(cudaEventRecord(done[c & 1], st));
        }
        if (c > 0) {
            FG_CUDA(cudaEventSynchronize(done[(c - 1) & 1]));
            if (!arena->live[(c - 1) & 1]) break;
        }
    }
    FG_CUDA(cudaStreamSynchronize(st));
    return FG_OK;
}

// whether a cycle is a graph, whose nodes hold the address of the flags
bool BatchRun::use_graph_streams(bool use_graph) const { return use_graph && P && P->bins.empty(); }

// Once members stopped: the remaining ones spread over all CTAs again, or move
// on chip now that they fit.  Nothing is in flight.
int BatchRun::reschedule(const std::vector<int> &live)
{
    int was = 0, now = 0;
    for (size_t i = 0; i < live.size(); ++i) {
        was += sched.empty() || sched[i];
        now += live[i];
    }
    if (now == was || now == 0) return FG_OK;
    sched = live;
    int r = choose_engine(mem, cfg, hs, live, P->B, st);
    if (r) return r;
    std::vector<CycItem> cyc;
    gang_items(hs, live, P->B, !cfg.mixed, cyc, P->bins);
    if (P->bins.empty()) return FG_OK;               // still streaming: nothing changed
    unsigned char *d = arena->dev.as<unsigned char>();
    auto put = [&](const Plan::Span &to, const void *from, size_t bytes) -> cudaError_t {
        unsigned char *h = arena->host + (to.as<unsigned char>() - d);
        std::memcpy(h, from, bytes);
        return cudaMemcpyAsync(to.p, h, bytes, cudaMemcpyHostToDevice, st);
    };
    FG_CUDA(put(P->sysdev, hs.data(), sizeof(SysDev) * hs.size()));
    FG_CUDA(put(P->cyc_items, cyc.data(), sizeof(CycItem) * cyc.size()));
    return FG_OK;
}

// True residual of the listed members' current x (FP64), then their state.
int BatchRun::finish(const std::vector<int> &idx, std::vector<SysState> &out)
{
    out.assign(idx.size(), SysState{});
    if (idx.empty()) return FG_OK;
    // every member: the run's own tables; some: tables of their own
    std::vector<BatchMember> sub;
    std::vector<SysDev> shs;
    const bool all = idx.size() == mem.size() && P;
    for (int i : idx) { sub.push_back(mem[i]); shs.push_back(hs[i]); }
    Plan F;
    PlanArena &ar = all ? *arena : sub_arena;
    if (!all) {
        int r = build_plan(F, sub, cfg, shs, false, sub_arena, st);
        if (r) return r;
    }
    const Plan &T = all ? *P : F;
    const SysDev *sys = T.sysdev.as<SysDev>();
    if (T.rprec) launch_elem_prec(sys, T.nsys, 3, 2, 0, st);   // pgmres.c:186: X = precondR(X)
    count_launches(enqueue_matvec<double>(T, 3, 0, st));
    k_final<<<grid_for(T.n_dch), kThreads, 0, st>>>(sys, T.dchunks.as<DChunk>(), T.dcount.as<int>());
    k_states<<<(T.nsys + 127) / 128, 128, 0, st>>>(sys, T.nsys, ar.states);
    FG_CUDA(cudaGetLastError());
    count_launches(2);
    FG_CUDA(cudaStreamSynchronize(st));
    for (size_t q = 0; q < idx.size(); ++q) out[q] = ar.states[all ? idx[q] : (int)q];
    return FG_OK;
}

// Drop members (indices ascending or not); the tables are rebuilt at the
// next commit().
void BatchRun::remove(std::vector<int> idx)
{
    std::sort(idx.rbegin(), idx.rend());
    for (int i : idx) {
        mem.erase(mem.begin() + i);
        hs.erase(hs.begin() + i);
    }
    if (exec) { cudaGraphExecDestroy(exec); exec = nullptr; }
    P.reset();
}

void fill_stats(const SysState &s, double secs, fg_solve_stats &o)
{
    o.iterations = s.iterations;
    o.cycles = s.cycles;
    o.converged = s.status == FG_ERR_TIMEOUT ? 0 : s.converged;   // (another CTA of its gang may have set it)
    o.status = s.status;
    o.rho = s.rho;
    o.eps = s.eps;
    o.true_rel_residual = s.true_res;
    o.seconds = secs;
}

static int run_batch(std::vector<BatchMember> &mem, const SolveConfig &cfg, fg_solve_stats *stats, cudaStream_t st)
{
    if (mem.empty()) return FG_OK;
    for (auto &m : mem) {
        int r = validate_member(m.s, cfg);
        if (r) return r;
    }
    auto t0 = std::chrono::steady_clock::now();
    BatchRun run(cfg, st, &mem[0].s->arena);
    int r;
    for (auto &m : mem)
        if ((r = run.stage(m))) return r;
    if ((r = run.commit()) || (r = run.run(cfg.use_graph != 0, cfg.lmax + 2))) return r;
    std::vector<int> all(mem.size());
    for (size_t i = 0; i < all.size(); ++i) all[i] = (int)i;
    std::vector<SysState> sts;
    if ((r = run.finish(all, sts))) return r;
    for (size_t i = 0; i < mem.size(); ++i) {
        BatchMember &m = mem[i];
        fg_system *sy = m.s;
        if (!m.X) continue;
        if (cfg.device_io) {
            FG_CUDA(cudaMemcpyAsync(m.X, sy->ws.x.p, 8 * (size_t)(sy->topo.n + 1), cudaMemcpyDeviceToDevice, st));
        } else {
            if ((r = permute_out(sy, sy->ws.x.as<double>(), sy->ws.r64.as<double>(), st))) return r;
            FG_CUDA(cudaMemcpyAsync(m.X, sy->ws.r64.p, 8 * (size_t)(sy->topo.n + 1), cudaMemcpyDeviceToHost, st));
        }
    }
    FG_CUDA(cudaStreamSynchronize(st));
    double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (stats)
        for (size_t i = 0; i < mem.size(); ++i) fill_stats(sts[i], secs, stats[i]);
    return FG_OK;
}

int solve_batch(std::vector<BatchMember> &mem, const SolveConfig &cfg, fg_solve_stats *stats, cudaStream_t st)
{
    const int r = run_batch(mem, cfg, stats, st);
    // copies from the caller's vectors and values of members whose own streams know nothing of st
    if (r) cudaStreamSynchronize(st);
    return r;
}

// Single matvec on device vectors (internal numbering, FP64 in/out).
int matvec_device(fg_system *s, const double *x, double *y, int precision, cudaStream_t st)
{
    if (!s->blocks_ok) { set_error("matvec before element blocks were set"); return FG_ERR_STATE; }
    const Topology &t = s->topo;
    if (precision == 32 && s->op != FG_OP_CSR) {
        int rb = ensure_blocks32(s, st);
        if (rb) return rb;
    }
    SysDev D{};
    D.n = t.n; D.n_pad = s->n_pad; D.nel = t.nel; D.nel_pad = s->nel_pad; D.S = t.S;
    D.lm = s->lm.as<int>(); D.A64 = s->A64.as<double>(); D.A32 = s->A32.as<float>();
    set_patch_fields(D, s);
    DevMem sd, ch, cnt;
    std::vector<EChunk> ech;
    std::vector<int> off(t.npcol + 1, 0), counts(t.npcol);
    for (int c = 0; c < t.npcol; ++c) {
        for (int q = t.pc_ptr[c]; q < t.pc_ptr[c + 1]; ++q) ech.push_back({0, t.pc_list[q], 0});
        off[c + 1] = (int)ech.size();
        counts[c] = off[c + 1] - off[c];
    }
    int r;
    if ((r = sd.alloc(sizeof(SysDev))) || (r = ch.alloc(sizeof(EChunk) * std::max<size_t>(1, ech.size()))) ||
        (r = cnt.alloc(sizeof(int) * std::max(1, t.npcol))))
        return r;
    FG_CUDA(cudaMemcpyAsync(sd.p, &D, sizeof(SysDev), cudaMemcpyHostToDevice, st));
    if (!ech.empty()) FG_CUDA(cudaMemcpyAsync(ch.p, ech.data(), sizeof(EChunk) * ech.size(), cudaMemcpyHostToDevice, st));
    if (t.npcol) FG_CUDA(cudaMemcpyAsync(cnt.p, counts.data(), sizeof(int) * t.npcol, cudaMemcpyHostToDevice, st));
    FG_CUDA(cudaMemsetAsync(y, 0, 8 * (size_t)(t.n + 1), st));
    if (s->op == FG_OP_CSR) {
        if ((r = csr_refresh(s, st))) return r;
        std::vector<DChunk> dch;
        for (int d = 0; d < t.n; d += 2048) dch.push_back({0, 0, d, std::min(d + 2048, t.n)});
        DevMem dc, dn;
        int nd = (int)dch.size();
        if ((r = dc.alloc(sizeof(DChunk) * std::max<size_t>(1, dch.size()))) || (r = dn.alloc(sizeof(int)))) return r;
        if (nd) FG_CUDA(cudaMemcpyAsync(dc.p, dch.data(), sizeof(DChunk) * nd, cudaMemcpyHostToDevice, st));
        FG_CUDA(cudaMemcpyAsync(dn.p, &nd, sizeof(int), cudaMemcpyHostToDevice, st));
        dim3 g = grid_for(std::max(nd, 1));
        const SysDev *sdp = sd.as<SysDev>();
        const DChunk *dcp = dc.as<DChunk>();
        const int *dnp = dn.as<int>();
        if (precision == 32) {
            if (s->csr_w == 4) k_csr_mv<4, float><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
            else if (s->csr_w == 8) k_csr_mv<8, float><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
            else k_csr_mv<32, float><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
        } else {
            if (s->csr_w == 4) k_csr_mv<4, double><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
            else if (s->csr_w == 8) k_csr_mv<8, double><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
            else k_csr_mv<32, double><<<g, kThreads, 0, st>>>(sdp, dcp, dnp, x, y);
        }
        FG_CUDA(cudaGetLastError());
        count_launches(1);
        FG_CUDA(cudaStreamSynchronize(st));
        return FG_OK;
    }
    for (int c = 0; c < t.npcol; ++c) {
        if (!counts[c]) continue;
        const EChunk *cp = ch.as<EChunk>() + off[c];
        const int *np = cnt.as<int>() + c;
        if (precision == 32)
            MvLaunch::go<float>(t.S, counts[c], st, sd.as<SysDev>(), cp, np, x, y, D.maxdof);
        else
            MvLaunch::go<double>(t.S, counts[c], st, sd.as<SysDev>(), cp, np, x, y, D.maxdof);
    }
    FG_CUDA(cudaGetLastError());
    count_launches(t.npcol);
    FG_CUDA(cudaStreamSynchronize(st));
    return FG_OK;
}

// The batched matvec alone, timed with CUDA events (fg_bench_matvec).
int bench_matvec(std::vector<fg_system *> &systems, int precision, int reps, double *ms, double *bytes)
{
    if (systems.empty() || reps < 1) { set_error("empty batch or reps < 1"); return FG_ERR_ARG; }
    SolveConfig cfg;
    cfg.mixed = precision == 32 ? 1 : 0;
    cfg.kmax = 2;
    std::vector<BatchMember> mem;
    std::vector<SysDev> hs;
    double b = 0;
    const double w = cfg.mixed ? 4.0 : 8.0;
    for (auto *s : systems) {
        if (!s->blocks_ok) { set_error("matvec before element blocks were set"); return FG_ERR_STATE; }
        int kk = std::max(2, s->ws.kmax);
        int r = ensure_workspace(s, kk, cfg.mixed);
        if (r || (r = rows_refresh(s, cfg.mixed != 0, systems[0]->stream))) return r;
        cfg.kmax = kk;
        mem.push_back({s, nullptr, nullptr, nullptr});
        hs.push_back(make_desc(s, cfg, false));
        const Topology &t = s->topo;
        // the assembled operator: values, columns, x once, y once
        b += (double)t.rw_col.size() * (t.ndof * t.ndof * w + (t.rw_dc.empty() ? 4.0 : 2.0)) + 2.0 * t.n * w;
    }
    cudaStream_t st = systems[0]->stream;
    Plan P;
    PlanArena arena;
    int r = build_plan(P, mem, cfg, hs, false, arena, st);
    if (r) return r;
    cudaEvent_t e0, e1;
    FG_CUDA(cudaEventCreate(&e0));
    FG_CUDA(cudaEventCreate(&e1));
    auto run = [&](int n) {
        for (int i = 0; i < n; ++i)
            count_launches(cfg.mixed ? enqueue_matvec<float>(P, 2, 0, st) : enqueue_matvec<double>(P, 2, 0, st));
    };
    run(2);  // warm-up
    cudaEventRecord(e0, st);
    run(reps);
    cudaEventRecord(e1, st);
    cudaError_t ce = cudaEventSynchronize(e1);
    float t = 0;
    if (ce == cudaSuccess) ce = cudaEventElapsedTime(&t, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (ce != cudaSuccess) return cuda_fail(ce, "bench_matvec");
    FG_CUDA(cudaStreamSynchronize(st));
    *ms = t / reps;
    *bytes = b;
    return FG_OK;
}

// Colour-by-colour matvec y += A x from a caller-placed descriptor and chunk
// table (device memory the caller owns); used by fg_matvec_noalloc.
int launch_matvec_colours(int S, int precision, const SysDev *sys_dev, const EChunk *ch_dev, const int *counts_dev,
                          const int *off_host, int ncol, int maxdof, const double *x, double *y, cudaStream_t st)
{
    for (int c = 0; c < ncol; ++c) {
        int cnt = off_host[c + 1] - off_host[c];
        if (!cnt) continue;
        const EChunk *cp = ch_dev + off_host[c];
        const int *np = counts_dev + c;
        if (precision == 32)
            MvLaunch::go<float>(S, cnt, st, sys_dev, cp, np, x, y, maxdof);
        else
            MvLaunch::go<double>(S, cnt, st, sys_dev, cp, np, x, y, maxdof);
        count_launches(1);
    }
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

static std::atomic<long long> g_launches{0};
void count_launches(long long n) { g_launches += n; }
long long launch_total() { return g_launches.load(); }

}  // namespace fg
