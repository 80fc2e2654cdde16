// The assembled operator of the Krylov engine: pattern by mesh unit, values
// summed from the element blocks on the device, and its matvec.
//
// GMRES applies the same operator hundreds of times between two builds, and
// that is bound by the bytes it reads.  Element by element a P1 mesh reads
// 2 S^2 values per node (two elements per node) plus their equation
// numbers, and scatters: one launch per patch colour, products staged and
// summed.  Assembled it is about 7 coupled nodes per node, B^2 values and one
// column each, summed by the thread that owns the row: one launch, no
// staging, no atomics.  Bytes per node and matvec, FP32 (FP64):
//   1 dof   105 (177) by elements,   50  (78) assembled
//   3 dofs  756 (1404),             290 (542)
//   4 dofs 1296 (2448),             494 (942)
// The same holds for the FP64 pipe (about 2 FMA per clock and SM on this
// part): 12 x 12 blocks take 288 FMA per node by elements, 112 assembled.
// The sums differ from the element order by rounding only; an FP32 entry is
// the FP64 sum rounded once.
// One matvec, by elements -> assembled (GB300, FP32 / FP64):
//   48 transport systems, 5.6 M dofs   119 -> 46 us / 427 -> 95 us
//   Euler 513 x 513 (4 dofs a node)    103 -> 43 us / 262 -> 82 us
//   Navier-Stokes 513 x 513 (3 dofs)    72 -> 25 us / 162 -> 70 us
// The values cost about one element matvec per solve.  A single matvec
// (fg_matvec, fg_matvec_noalloc) stays with the element blocks.
//
// Layout: units (1 dof per node: the internal dofs; else the mesh nodes) in
// slices of kRowSlice; slot k of unit l of a slice starts at entry
// e = off[slice] + k * kRowSlice + l: its column (a unit) at col[e], the
// column's distance from the unit at dc[e] where 16 bits hold all of them, its
// B x B block, row-major, at value e * B * B.  A slice is as wide as its
// widest unit, or, where that pads by an eighth at most, as the widest of all.
// Rows and columns of prescribed dofs are zero.
#include <algorithm>
#include <type_traits>

#include <cuda_fp16.h>

#include "system.h"

namespace fg {

// ---------------------------------------------------------------- values
// One thread per (unit, row): for every slot the contributions of the unit's
// elements, in reference element order.  Reads A64 once (8 S^2 bytes per
// element), writes the values once; runs once per solve.
template <int B, bool F32>
__global__ void __launch_bounds__(256)
k_rows_values(int nunits, int n, const int *__restrict__ off, const int *__restrict__ col, const int *__restrict__ inc_ptr,
              const int *__restrict__ inc, const int *__restrict__ vert, const int *__restrict__ node_dof,
              const double *__restrict__ A64, int ld, double *__restrict__ v64, float *__restrict__ v32)
{
    constexpr int S = 3 * B, BITS = B == 1 ? 4 : 2;      // dof incidence pos * 16 + row, node incidence pos * 4 + vertex
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int ns = (nunits + kRowSlice - 1) / kRowSlice;
    const int u = (int)(t / B), r = (int)(t - (long long)u * B);
    if (u >= ns * kRowSlice) return;
    const int s = u / kRowSlice, l = u % kRowSlice;
    const bool live = u < nunits && (B == 1 || node_dof[u * B + r] != n);
    const int q0 = u < nunits ? inc_ptr[u] : 0, q1 = u < nunits ? inc_ptr[u + 1] : 0;
    for (int e = off[s] + l; e < off[s + 1]; e += kRowSlice) {
        const int m = col[e];
        double a[B];
#pragma unroll
        for (int c = 0; c < B; ++c) a[c] = 0.0;
        if (live && m >= 0) {
            for (int q = q0; q < q1; ++q) {
                const int v = inc[q], pos = v >> BITS, i = v & ((1 << BITS) - 1);
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    if (vert[(size_t)b * ld + pos] != m) continue;
                    const double *src = A64 + (size_t)((B * i + r) * S + B * b) * ld + pos;
#pragma unroll
                    for (int c = 0; c < B; ++c) a[c] += src[(size_t)c * ld];
                }
            }
            if (B > 1) {
#pragma unroll
                for (int c = 0; c < B; ++c)
                    if (node_dof[m * B + c] == n) a[c] = 0.0;
            }
        }
        const size_t o = ((size_t)e * B + r) * B;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            v64[o + c] = a[c];
            if (F32) v32[o + c] = (float)a[c];
        }
    }
}

static size_t rows_entries(const fg_system *s) { return s->topo.rw_col.size() * (size_t)(s->topo.ndof * s->topo.ndof); }

size_t rows_bytes(const fg_system *s, bool fp32)
{
    const size_t ne = rows_entries(s);
    return (s->rw64.p ? 0 : 8 * ne) + (fp32 && !s->rw32.p ? 4 * ne : 0);
}

int rows_refresh(fg_system *s, bool fp32, cudaStream_t st)
{
    if (s->rw64_ok && (!fp32 || s->rw32_ok)) return FG_OK;
    if (!s->blocks_ok) { set_error("assembled operator needs element blocks"); return FG_ERR_STATE; }
    const Topology &t = s->topo;
    const size_t ne = rows_entries(s);
    int r;
    if (!s->rw64.p && (r = s->rw64.alloc(8 * ne))) return r;
    if (fp32 && !s->rw32.p && (r = s->rw32.alloc(4 * ne))) return r;
    const int ns = (t.nunits + kRowSlice - 1) / kRowSlice;
    if (ns > 0) {
        const int *ip = t.ndof == 1 ? s->dinc_ptr.as<int>() : s->ninc_ptr.as<int>();
        const int *in = t.ndof == 1 ? s->dinc.as<int>() : s->ninc.as<int>();
        const int *vx = t.ndof == 1 ? s->lm.as<int>() : s->gien.as<int>();
        const long long nt = (long long)ns * kRowSlice * t.ndof;
        const unsigned g = (unsigned)((nt + 255) / 256);
        auto go = [&](auto b, auto f) {
            k_rows_values<decltype(b)::value, decltype(f)::value><<<g, 256, 0, st>>>(
                t.nunits, t.n, s->rw_off.as<int>(), s->rw_col.as<int>(), ip, in, vx, s->node_dof.as<int>(),
                s->A64.as<double>(), s->nel_pad, s->rw64.as<double>(), s->rw32.as<float>());
        };
        auto with = [&](auto b) { if (fp32) go(b, std::true_type{}); else go(b, std::false_type{}); };
        switch (t.ndof) {
        case 1: with(std::integral_constant<int, 1>{}); break;
        case 2: with(std::integral_constant<int, 2>{}); break;
        case 3: with(std::integral_constant<int, 3>{}); break;
        case 4: with(std::integral_constant<int, 4>{}); break;
        }
        FG_CUDA(cudaGetLastError());
        count_launches(1);
    }
    s->rw64_ok = true;
    if (fp32) s->rw32_ok = true;
    return FG_OK;
}

// ---------------------------------------------------------------- matvec
template <typename TA, typename TX> __device__ __forceinline__ TA row_x(TX v, const SysDev &D)
{
    if constexpr (std::is_same<TX, __half>::value) return (TA)(__half2float(v) * D.vsci);
    else return (TA)v;
}
// one block row of B values (16-byte loads for B = 2, 4)
template <int B, typename T> __device__ __forceinline__ void row_vals(const T *p, T (&a)[B])
{
    if constexpr (B == 1) a[0] = __ldcs(p);
    else if constexpr (B == 4 && sizeof(T) == 4) {
        const float4 v = __ldcs(reinterpret_cast<const float4 *>(p));
        a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
    } else if constexpr (B % 2 == 0 && sizeof(T) == 8) {
#pragma unroll
        for (int c = 0; c < B; c += 2) {
            const double2 v = __ldcs(reinterpret_cast<const double2 *>(p + c));
            a[c] = v.x;
            a[c + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < B; ++c) a[c] = __ldg(p + c);
    }
}
// one unit's B dof numbers
template <int B> __device__ __forceinline__ void unit_dofs(const int *nd, int u, int (&d)[B])
{
    if constexpr (B == 1) d[0] = u;
    else if constexpr (B == 4) {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(nd) + u);
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    } else {
#pragma unroll
        for (int c = 0; c < B; ++c) d[c] = __ldg(nd + (size_t)u * B + c);
    }
}

// y = A x, a thread per (unit, row), 32 / B units per warp (so that a
// node's rows are in one warp: BlockDiag is applied by shuffles).  HBM-bound;
// every slot's loads are independent, four to eight in flight per thread.
// out 2 fuses M^-1 into the store, so the Arnoldi pass that follows reads
// w as it is.
template <int B, typename TA, typename TX>
__global__ void __launch_bounds__(kThreads)
k_rows_mv(const SysDev *__restrict__ sys, const NChunk *__restrict__ ch, const int *__restrict__ nch, int gate,
          int in_sel, int out, int step)
{
    constexpr int UW = 32 / B, UC = UW * (kThreads / 32);
    constexpr int U = B == 1 ? 8 : 4;
    const int total = *nch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lu = lane / B, r = lane - lu * B;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const NChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!(gate < 0 || (gate == 0 ? D.st->live != 0 : D.st->in_cycle != 0))) continue;
        const TX *X = in_sel == 0 ? (const TX *)D.x
                    : in_sel == 1 ? (const TX *)D.V + (size_t)step * D.n_pad : (const TX *)D.r64;
        const TA *A = sizeof(TA) == 8 ? (const TA *)D.rw64 : (const TA *)D.rw32;
        const int n = D.n;
        const int *col = D.rw_col, *nd = D.node_dof;
        const short *dc = D.rw_dc;
        const int ru = D.rw_u;
        if constexpr (B == 1 && sizeof(TA) == 4) {
            // Slices of one width, at most U: two rows a thread, in 8- and 4-byte
            // loads.  The pass waits on its loads: half the instructions carry the
            // same bytes, and 1.7 times the rows are in flight (4.0 M dofs:
            // one row a thread and 32-bit columns 63 us, 16-bit and twice the
            // CTAs 52, two rows 38; 33 at copy bandwidth).
            if (dc && ru > 0 && ru <= U) {
                for (int u = k.n0 + 2 * threadIdx.x; u < k.n1; u += 2 * kThreads) {
                    const bool two = u + 1 < k.n1;
                    const int e = u / kRowSlice * ru * kRowSlice + u % kRowSlice;
                    short2 m[U];
                    float2 a[U];
#pragma unroll
                    for (int q = 0; q < U; ++q) {
                        m[q] = make_short2(0, 0);
                        a[q] = make_float2(0.0f, 0.0f);
                        if (q < ru) {
                            m[q] = __ldcs(reinterpret_cast<const short2 *>(dc + e + q * kRowSlice));
                            a[q] = __ldcs(reinterpret_cast<const float2 *>(A + e + q * kRowSlice));
                        }
                    }
                    const float2 pc = out == 2 && D.precond == FG_PRECOND_DIAG
                                          ? make_float2(((const float *)D.invd32)[u], ((const float *)D.invd32)[two ? u + 1 : u])
                                          : make_float2(1.0f, 1.0f);
                    float x0[U], x1[U], y0 = 0.0f, y1 = 0.0f;
#pragma unroll
                    for (int q = 0; q < U; ++q) {
                        x0[q] = row_x<TA, TX>(X[u + m[q].x], D);
                        x1[q] = row_x<TA, TX>(X[two ? u + 1 + m[q].y : u], D);
                    }
#pragma unroll
                    for (int q = 0; q < U; ++q) { y0 += a[q].x * x0[q]; y1 += a[q].y * x1[q]; }
                    y0 *= pc.x;
                    y1 *= pc.y;
                    if (out == 0) {
                        D.t64[u] = (double)y0;
                        if (two) D.t64[u + 1] = (double)y1;
                    } else {
                        float *o = (float *)(out == 2 ? D.w : D.t);
                        if (two) *reinterpret_cast<float2 *>(o + u) = make_float2(y0, y1);
                        else o[u] = y0;
                    }
                }
                continue;
            }
        }
        for (int u0 = k.n0; u0 < k.n1; u0 += UC) {
            const int u = u0 + warp * UW + lu;
            const bool on = lu < UW && u < k.n1;
            TA y = (TA)0;
            int id = n;
            if (on) {
                id = B == 1 ? u : nd[(size_t)u * B + r];
                const int s = u / kRowSlice;
                const int e0 = ru ? s * ru * kRowSlice : __ldg(D.rw_off + s), e1 = ru ? e0 + ru * kRowSlice : __ldg(D.rw_off + s + 1);
                for (int e = e0 + u % kRowSlice; e < e1; e += U * kRowSlice) {
                    int m[U];
                    TA a[U][B], x[U][B];
                    if (dc) {
#pragma unroll
                        for (int q = 0; q < U; ++q) m[q] = e + q * kRowSlice < e1 ? __ldcs(dc + e + q * kRowSlice) : 0;
                    } else {
#pragma unroll
                        for (int q = 0; q < U; ++q) m[q] = e + q * kRowSlice < e1 ? (__ldcs(col + e + q * kRowSlice) & ~kRowPad) - u : 0;
                    }
#pragma unroll
                    for (int q = 0; q < U; ++q)
                        if (e + q * kRowSlice < e1) row_vals<B, TA>(A + ((size_t)(e + q * kRowSlice) * B + r) * B, a[q]);
                        else
#pragma unroll
                            for (int w = 0; w < B; ++w) a[q][w] = (TA)0;
#pragma unroll
                    for (int q = 0; q < U; ++q) {
                        int d[B];
                        unit_dofs<B>(nd, u + m[q], d);
#pragma unroll
                        for (int w = 0; w < B; ++w) x[q][w] = row_x<TA, TX>(X[d[w]], D);
                    }
#pragma unroll
                    for (int q = 0; q < U; ++q)
                    {
                        TA z = a[q][0] * x[q][0];     // the block's product first: short chains
#pragma unroll
                        for (int w = 1; w < B; ++w) z += a[q][w] * x[q][w];
                        y += z;
                    }
                }
            }
            if (out == 2) {
                if (B > 1 && D.precond == FG_PRECOND_BLOCKDIAG) {
                    const TA *M = (sizeof(TA) == 8 ? (const TA *)D.ibd64 : (const TA *)D.ibd32);
                    TA m[B], z = (TA)0;
                    if (on) row_vals<B, TA>(M + ((size_t)u * B + r) * B, m);
                    if (id == n) y = (TA)0;
#pragma unroll
                    for (int q = 0; q < B; ++q) {
                        const TA yq = __shfl_sync(0xffffffffu, y, min(lu * B + q, 31));
                        z = q == 0 ? m[0] * yq : z + m[q] * yq;
                    }
                    y = z;
                } else if (D.precond == FG_PRECOND_DIAG && on && id != n) {
                    y *= sizeof(TA) == 8 ? ((const TA *)D.invd64)[id] : ((const TA *)D.invd32)[id];
                }
                if (on && id != n) ((TA *)D.w)[id] = y;
            } else if (on && id != n) {
                if (out == 0) D.t64[id] = (double)y;
                else ((TA *)D.t)[id] = y;
            }
        }
    }
}

template <int B>
static void rows_mv(int prec, dim3 g, const SysDev *sys, const NChunk *ch, const int *nch, int gate, int in_sel, int out,
                    int step, cudaStream_t st)
{
    if (prec == 64) k_rows_mv<B, double, double><<<g, kThreads, 0, st>>>(sys, ch, nch, gate, in_sel, out, step);
    else if (prec == 32) k_rows_mv<B, float, float><<<g, kThreads, 0, st>>>(sys, ch, nch, gate, in_sel, out, step);
    else k_rows_mv<B, float, __half><<<g, kThreads, 0, st>>>(sys, ch, nch, gate, in_sel, out, step);
}

int launch_rows_mv(int B, int prec, const SysDev *sys, const NChunk *ch, const int *nch, int nchunks, int gate,
                   int in_sel, int out, int step, cudaStream_t st)
{
    const dim3 g((unsigned)std::max(1, std::min(nchunks, 16 * sm_count())));
    switch (B) {
    case 1: rows_mv<1>(prec, g, sys, ch, nch, gate, in_sel, out, step, st); break;
    case 2: rows_mv<2>(prec, g, sys, ch, nch, gate, in_sel, out, step, st); break;
    case 3: rows_mv<3>(prec, g, sys, ch, nch, gate, in_sel, out, step, st); break;
    case 4: rows_mv<4>(prec, g, sys, ch, nch, gate, in_sel, out, step, st); break;
    }
    return 1;
}

}  // namespace fg
