// One restart cycle of GMRES on chip: the Arnoldi steps of a system as one
// persistent gang of CTAs that holds the Krylov basis in shared memory.
//
// Why.  As one kernel per pass an Arnoldi step of the systems served here (1k
// to 260k equations) is launch and latency bound: 30 to 80 us for work that
// the chip's shared memory does in 1 or 2.  The basis of a whole restart
// cycle fits it: 152 SMs x 227 KB hold 30 vectors of 276k FP32 (138k FP64)
// entries.  So a gang of g CTAs (one per SM) owns a system for a cycle, CTA
// `rank` the units [u0, u1) and their rows of every basis vector, and keeps
// as many of their operator rows beside them as fit; the other rows are read
// from L2 each step, and only the newest vector and the reductions pass
// between CTAs.
//
// A step (classical Gram-Schmidt with a Gram correction: with G = V^T V the
// coefficients of the two classical passes are s + (s - G s), s = V^T w, so
// one pass over the basis gives both; FP64 systems too).  The newest vector
// is kept unscaled until its norm is known (but for a power of two that a cycle's
// first step finds, unit_scale), so that the norm travels with the next step's
// dots and a step has a single reduction over the gang:
//   1. the Gram column V^T v_i over the CTA's rows, 8 lanes per basis vector,
//      while the newest vector's entries of neighbouring CTAs (the halo)
//      arrive: polled from the exchange vector vb into shared memory;
//   2. w = M^-1 A v_i for the CTA's rows;
//   3. s = V^T w; exchange: both and ||v_i||^2 summed over the gang;
//   4. v_i and w scaled by 1 / ||v_i||, c = s - (G - I) s, w -= V c; the
//      entries that neighbours need go to vb.
// The Givens rotations of column i - 1 run in a warp of their own on rank 0
// while step i goes on; a stop is announced with the exchange of step i + 1, so
// up to two steps of a cycle that ends early are wasted.
//
// Exchanges carry their own flags: every 32 bits are stored with the step's
// tag as one 64-bit word, and readers poll for the tag, so an exchange costs
// one trip through L2 (small gangs: every CTA sums all partials; vb) or two
// (large gangs: CTA m sums slot m, everyone reads the totals) and no barrier
// or fence.  Partials are summed in rank order: results are the same run to
// run, and depend on the gang only through its size (gang_size: the system's, or
// in larger batches the room's too).  A word is rewritten only after every CTA published the
// exchange that follows its reading.
//
// Measured (GB300), a whole solve with the pass kernels -> on chip, and an
// Arnoldi step: 961 equations FP64 8.8 -> 2.0 ms (6 us a step), 16k FP64 26.5 ->
// 6.3 ms (7 us), 16k FP32 21.9 -> 4.5 ms (5 us), 261k FP32 94 -> 27 ms (9.5 us).
// (The same build differs by up to 8 % between processes and machines.)
// What is left of a step is mostly the two trips through L2 of the exchange
// (2 to 5 us with the CTAs' skew); the basis sweeps take 2 to 3 us.
//
// FP32 systems keep FP64 out of the steps: this part's FP64 pipe issues one
// warp instruction in 16 cycles, so sums across CTAs are error-free FP32
// pairs.
//
// The launch is cooperative, so all CTAs are resident; a CTA is one rank of
// one system's gang.  Polls are bounded (~2 s, or the number fg_set_wait_limit
// gives): a CTA that gives up marks the system FG_ERR_TIMEOUT and leaves at the
// step's next barrier, all its threads together.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "sums.cuh"

namespace fg {

namespace {

// Threads per CTA besides the Givens warp, one CTA an SM.  Halving the ranks
// halves the words that a reduction polls, and the rank with a whole SM's rows
// keeps as many threads: 148k equations FP64 38.8 -> 33.7 ms a solve (two CTAs of
// 256 -> one of 512), 263k FP32 31.7 -> 24.1, 16k FP32 4.9 -> 4.2; one of 384
// 36.9, 28.3, 4.5 (where 512 took 35.7, 26.4, 4.3), one of 256 39.0, 31.8, 4.4.
constexpr int kWorkers = 512;
constexpr int kCycThreads = kWorkers + 32;
constexpr int kGroups = kWorkers / 8;         // 8-lane groups
constexpr int kMaxSlices = 8;
static_assert(kMaxRestart <= kGroups, "a group for every basis vector");
// slices of the CTA's rows in the dots: while every lane keeps 8 packs
__device__ __forceinline__ int dot_slices(int np, int nv) { return max(1, min(min(kMaxSlices, np / 64), kGroups / nv)); }
constexpr long long kPollCycles = 4000000000LL;   // ~2 s
__device__ int g_gang_polls = 1 << 24;            // fg_set_wait_limit
// gangs up to this size sum all partials in every CTA (16k equations FP32 in the
// 32 CTAs of an earlier row count, 64 now: 5.3 ms a solve in two trips, 6.4 in one)
constexpr int kDirect32 = 8, kDirect64 = 8;

template <typename T> struct Pack { static constexpr int N = 16 / sizeof(T); };
template <typename T, int N> struct alignas(16) Vec { T v[N]; };
template <typename T> __device__ __forceinline__ Vec<T, Pack<T>::N> ldp(const T *p)
{
    return *reinterpret_cast<const Vec<T, Pack<T>::N> *>(p);
}

// ---------------------------------------------------------------- exchange
typedef unsigned long long u64;
__device__ __forceinline__ u64 word(unsigned v, unsigned tag) { return ((u64)tag << 32) | v; }
__device__ __forceinline__ void put1(u64 *p, unsigned v, unsigned tag)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(word(v, tag)) : "memory");
}
__device__ __forceinline__ void put2(u64 *p, unsigned v0, unsigned v1, unsigned tag)
{
    put1(p, v0, tag);
    put1(p + 1, v1, tag);
}
__device__ __forceinline__ u64 peek(const u64 *p)
{
    u64 w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(w) : "l"(p) : "memory");
    return w;
}
// The values of NW words p[k * stride], k < cnt, once each carries the tag.
// All loads of a round are in flight together.  Gives up after ~2 s or `polls`
// rounds, looked at every 32 (limits below that: every) rounds, or when the CTA
// already did (values are then garbage).
struct Bound {
    volatile int *gave_up;
    int mask;
};
template <int NW>
__device__ __forceinline__ void poll(const u64 *p, size_t stride, int cnt, unsigned tag, unsigned (&v)[NW],
                                     const Bound &bound)
{
    u64 w[NW];
    const long long t0 = clock64();
    for (int it = 0;; ++it) {
        bool ok = true;
#pragma unroll
        for (int k = 0; k < NW; ++k) w[k] = k < cnt ? peek(p + k * stride) : word(0u, tag);
#pragma unroll
        for (int k = 0; k < NW; ++k) ok = ok && (unsigned)(w[k] >> 32) == tag;
        if (ok) break;
        if ((it & bound.mask) == bound.mask && (*bound.gave_up || it + 1 >= g_gang_polls || clock64() - t0 > kPollCycles)) {
            *bound.gave_up = 1;
            break;
        }
    }
#pragma unroll
    for (int k = 0; k < NW; ++k) v[k] = (unsigned)w[k];
}
// a T as 32-bit words (FP32: 1, FP64: 2)
template <typename T> constexpr int kWords = sizeof(T) / 4;
template <typename T> __device__ __forceinline__ void put(u64 *p, T v, unsigned tag)
{
    if constexpr (sizeof(T) == 8) {
        const long long b = __double_as_longlong(v);
        put2(p, (unsigned)b, (unsigned)(b >> 32), tag);
    } else put1(p, __float_as_uint(v), tag);
}
template <typename T> __device__ __forceinline__ T from_words(const unsigned *v)
{
    if constexpr (sizeof(T) == 8) return __longlong_as_double(((long long)v[1] << 32) | v[0]);
    else return __uint_as_float(v[0]);
}

// a sum as two words of the exchange
__device__ __forceinline__ void put_pair(u64 *p, const Sum<double> &t, unsigned tag) { put<double>(p, t.h, tag); }
__device__ __forceinline__ void put_pair(u64 *p, const Sum<float> &t, unsigned tag)
{
    put2(p, __float_as_uint(t.h), __float_as_uint(t.l), tag);
}
__device__ __forceinline__ void add_pair(Sum<double> &t, const unsigned *v) { t.add(from_words<double>(v)); }
__device__ __forceinline__ void add_pair(Sum<float> &t, const unsigned *v)
{
    t.add(__uint_as_float(v[0]));
    t.l = __fadd_rn(t.l, __uint_as_float(v[1]));
}

// ---------------------------------------------------------------- rows
template <int B, typename T> __device__ __forceinline__ void load_vals(const T *p, T (&a)[B])
{
    if constexpr (B * sizeof(T) % 16 == 0) {
#pragma unroll
        for (int c = 0; c < B; c += Pack<T>::N) {
            const uint4 r = __ldg(reinterpret_cast<const uint4 *>(p + c));
            Vec<T, Pack<T>::N> v;
            memcpy(&v, &r, 16);
#pragma unroll
            for (int k = 0; k < Pack<T>::N; ++k) a[c + k] = v.v[k];
        }
    } else {
#pragma unroll
        for (int c = 0; c < B; ++c) a[c] = __ldg(p + c);
    }
}
// one unit of the newest vector, from shared memory
template <int B, typename T> __device__ __forceinline__ void load_x(const T *p, T (&a)[B])
{
    if constexpr (B * sizeof(T) % 16 == 0) {
#pragma unroll
        for (int c = 0; c < B; c += Pack<T>::N) {
            const auto v = ldp(p + c);
#pragma unroll
            for (int k = 0; k < Pack<T>::N; ++k) a[c + k] = v.v[k];
        }
    } else {
#pragma unroll
        for (int c = 0; c < B; ++c) a[c] = p[c];
    }
}

// The newest vector as a CTA holds it: its own units [u0, u1) in their basis
// slot, the halo [lo, u0), [u1, hi) behind one another.  A unit's local number
// counts its own units first.
template <typename T> struct Newest {
    const T *own, *halo;
    int u0, u1, lo;
    __device__ __forceinline__ int local(int m) const
    {
        return (unsigned)(m - u0) < (unsigned)(u1 - u0) ? m - u0 : m < u0 ? u1 - u0 + m - lo : m - lo;
    }
    template <int B> __device__ __forceinline__ const T *at(int l) const
    {
        return (l < u1 - u0 ? own : halo - (u1 - u0) * B) + l * B;
    }
};

// y + a . x, the same roundings wherever the row is kept
template <int B, typename T> __device__ __forceinline__ T row_add(T y, const T (&a)[B], const T (&x)[B])
{
    if constexpr (B == 1) return fma(a[0], x[0], y);
    T z = a[0] * x[0];
#pragma unroll
    for (int c = 1; c < B; ++c) z = fma(a[c], x[c], z);
    return y + z;
}

// A row of the operator from global memory times the newest vector: 16-bit
// columns, no slice offset where slices have one width (263k equations FP32, a
// fifth of the rows on chip: 26.2 -> 25.7 ms a solve; rows in pairs 26.3).
template <int B, typename T>
__device__ __forceinline__ T row_times_x(const int *__restrict__ off, const short *__restrict__ dc, int ru,
                                         const T *__restrict__ A, const Newest<T> &x, int u, int r)
{
    constexpr int U = B == 1 ? 8 : 4;
    const int s = u / kRowSlice, e0 = ru ? s * ru * kRowSlice : __ldg(off + s), e1 = ru ? e0 + ru * kRowSlice : __ldg(off + s + 1);
    T y = (T)0;
    for (int e = e0 + u % kRowSlice; e < e1; e += U * kRowSlice) {
        int m[U];
        T a[U][B];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const bool in = e + q * kRowSlice < e1;
            m[q] = in ? u + __ldg(dc + e + q * kRowSlice) : u;
            if (in) load_vals<B, T>(A + ((size_t)(e + q * kRowSlice) * B + r) * B, a[q]);
            else
#pragma unroll
                for (int c = 0; c < B; ++c) a[q][c] = (T)0;
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            T v[B];
            load_x<B, T>(x.template at<B>(x.local(m[q])), v);
            y = row_add<B, T>(y, a[q], v);
        }
    }
    return y;
}

__device__ __forceinline__ void sync_workers() { asm volatile("bar.sync 1, %0;\n" ::"n"(kWorkers) : "memory"); }

// 1 / sqrt(n2) in T
__device__ __forceinline__ float inv_norm(const Sum<float> &n2) { return rsqrtf(n2.rounded()); }
__device__ __forceinline__ double inv_norm(const Sum<double> &n2) { return rsqrt(n2.h); }
// sc^2 n2 - 1: the newest vector's Gram diagonal less 1
__device__ __forceinline__ float gram_diag(const Sum<float> &n2, float sc)
{
    const float p = __fmul_rn(sc, n2.h), e = __fmaf_rn(sc, n2.h, -p);
    return __fadd_rn(__fmaf_rn(p, sc, -1.f), __fmaf_rn(e, sc, n2.l * sc * sc));
}
__device__ __forceinline__ double gram_diag(const Sum<double> &n2, double sc) { return fma(sc * n2.h, sc, -1.0); }

// ---------------------------------------------------------------- the cycle
// SPILL: a system alone on the GPU whose basis passes its shared memory by up
// to a few times: the older basis vectors stay in shared memory, the others in
// global memory (L2), where only the CTA that owns the rows reads them; the two
// newest vectors have shared-memory slots of their own.
template <typename T, int B, bool SPILL>
__global__ void __launch_bounds__(kCycThreads, 1)
k_cycle(const SysDev *__restrict__ sys, const CycItem *__restrict__ items, int smem)
{
    constexpr int N = Pack<T>::N, KM = kMaxRestart + 4, WP = kWords<T>;
    extern __shared__ __align__(16) unsigned char cyc_smem[];
    T *V = reinterpret_cast<T *>(cyc_smem);
    __shared__ double s_cs[KM], s_sn[KM], s_g[KM + 1], s_t[KM], s_a[KM];
    __shared__ T s_tot[2 * KM], s_red[2 * KM], s_c[2][KM];     // c of this and the previous step
    __shared__ T s_n2h[kWorkers / 32], s_n2l[kWorkers / 32];
    __shared__ T s_sc, s_dg;                      // 1 / norm of the newest vector, its Gram diagonal less 1
    __shared__ T s_sg, s_ss;                      // the newest vector's power of two, times s_sc
    __shared__ int s_stop, s_gave_up, s_m;
    const Bound bound{&s_gave_up, g_gang_polls < 32 ? 0 : 31};
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l8 = tid & 7, gid = tid >> 3;
    const bool worker = tid < kWorkers;
    if (tid == 0) s_gave_up = 0;

    {
        const CycItem k = items[blockIdx.x];
        const SysDev &D = sys[k.sys];
        if (!D.st->in_cycle) return;
        const int km = D.kmax, rank = k.rank, g = D.cy_g, Rp = D.cy_rows, n = D.n;
        const int nrow = (k.u1 - k.u0) * B, np = Rp / N;
        const unsigned base = *D.cy_epoch;
        const T *A = sizeof(T) == 8 ? (const T *)D.rw64 : (const T *)D.rw32;
        // exchange words, by step parity where a CTA may publish the next step's while a
        // slower one still reads this step's
        u64 *const part2 = D.cy_part;                        // [parity][slot][rank], WP words each
        u64 *const norm2 = part2 + (size_t)4 * km * g * WP;  // [parity][rank], 2 words
        u64 *const total = norm2 + 4 * (size_t)g;            // [slot], WP words; the norm's 2 words
        u64 *const note = total + (size_t)2 * km * WP + 2;   // stop flag [parity], m, y [km][2]
        u64 *vb = (u64 *)D.cy_vb;                            // [row], WP words
        const int js = SPILL ? D.cy_js : km;                 // basis vectors in shared memory
        T *const W2 = V + (size_t)js * Rp;                   // SPILL: the two newest vectors
        T *const gV = SPILL ? (T *)D.cy_spill + (size_t)rank * Rp : nullptr;
        const size_t gs = (size_t)g * Rp;
        auto slot = [&](int j) -> T * { return !SPILL || j < js ? V + (size_t)j * Rp : gV + (j - js) * gs; };
        T *E = W2 + (SPILL ? 2 * (size_t)Rp : 0);             // Gram matrix less I, km x km
        T *halo = E + ((km * km + N - 1) & ~(N - 1));
        const bool direct = g <= (sizeof(T) == 8 ? kDirect64 : kDirect32);
        const int pre = D.precond;
        const double target = D.mixed ? D.st->target : D.st->eps;
        Rot R{s_cs, s_sn, s_g, s_t, s_a, 0, 0, 0, 0.0};
        const int lo = max(k.u0 - D.rw_lo, 0), hi = min(k.u1 + D.rw_hi, D.nunits);
        const int nhl = (k.u0 - lo) * B, nh = nhl + (hi - k.u1) * B;
        Newest<T> X{SPILL ? W2 : V, halo, k.u0, k.u1, lo};
        // rows [0, nc) of the operator: values [slot][row][B], local units [slot][row]
        const int W = D.rw_w;
        T *rv = halo + ((nh + N - 1) & ~(N - 1));
        const int nc = max(0, min(nrow, (int)((smem - (int)((unsigned char *)rv - cyc_smem)) / (max(W, 1) * (int)(B * sizeof(T) + 2))) & ~7));
        unsigned short *ri = reinterpret_cast<unsigned short *>(rv + (size_t)W * nc * B);
        const int *off = D.rw_off, *nd = D.node_dof;
        const short *dc = D.rw_dc;
        const int ru = D.rw_u;
        const T *M = B > 1 && pre == FG_PRECOND_BLOCKDIAG ? (sizeof(T) == 8 ? (const T *)D.ibd64 : (const T *)D.ibd32)
                   : pre == FG_PRECOND_DIAG ? (sizeof(T) == 8 ? (const T *)D.invd64 : (const T *)D.invd32) : nullptr;

        if (worker) {
            for (int q = tid; q < nc; q += kWorkers) {
                const int u = k.u0 + q / B, r = q % B, s = u / kRowSlice;
                const int e0 = __ldg(off + s) + u % kRowSlice, e1 = __ldg(off + s + 1);
                for (int w = 0; w < W; ++w) {
                    const int e = e0 + w * kRowSlice;
                    const int m = e < e1 ? u + __ldg(dc + e) : u;
                    T a[B];
                    if (e < e1) load_vals<B, T>(A + ((size_t)e * B + r) * B, a);
#pragma unroll
                    for (int c = 0; c < B; ++c) rv[((size_t)w * nc + q) * B + c] = e < e1 ? a[c] : (T)0;
                    ri[w * nc + q] = (unsigned short)X.local(m);
                }
            }
            // v_0 = r / ||r||, halo included
            const double sc = 1.0 / D.st->r0;
            auto v0 = [&](int row) -> T {
                const int id = B == 1 ? row : __ldg(nd + row);
                return id == n ? (T)0 : (T)(sc * D.r64[id]);
            };
            Sum<T> t;
            for (int q = tid; q < Rp; q += kWorkers) {
                const T v = q < nrow ? v0(k.u0 * B + q) : (T)0;
                (SPILL ? W2 : V)[q] = v;
                t.add_square(v);
            }
            for (int q = tid; q < nh; q += kWorkers) {
                halo[q] = v0(lo * B + (q < nhl ? q : q + nrow));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t.fold(o);
            if (lane == 0) {
                s_n2h[warp] = t.h;
                if constexpr (sizeof(T) == 4) s_n2l[warp] = t.l;
            }
            if (tid == 0) { s_stop = 0; s_g[0] = D.g[0]; }
        }
        __syncthreads();
        int i = 0;
        for (; i < km - 1; ++i) {
            const int nv = i + 1;
            const unsigned tag = base + (unsigned)i + 1u;
            u64 *part = part2 + (i & 1) * ((size_t)2 * km * g * WP), *norm = norm2 + (i & 1) * (2 * (size_t)g);
            T *vi = SPILL ? W2 + (i & 1) * Rp : V + (size_t)i * Rp;
            T *w = SPILL ? W2 + ((i + 1) & 1) * Rp : vi + Rp;
            X.own = vi;
            if (worker) {
                const int nsl = dot_slices(np, nv);
                // nsl groups a basis vector; FP32: a lane's eight chains, the lanes and the
                // slices are added in pairs (rms error of <v, w>, unit vectors, 500 emulated:
                // 961 rows 1.6e-9, 16k 4.2e-10, 261k 1.4e-10; four chains 2.0, 5.0, 1.6; FP32
                // folds 2.9, 7.4, 2.5; sequential chains with FP64 sums over warps 1.7, 4.2, 2.0)
                auto dot = [&](const T *y, T *red) {
                    if (gid - (gid & 3) >= nv * nsl) return;      // a warp without a vector
                    const int j = gid % nv, sl = gid / nv;
                    constexpr int H = sizeof(T) == 4 ? 2 : 1;      // FP32: two chains a lane and entry of a pack
                    T s4[H * N];
#pragma unroll
                    for (int c = 0; c < H * N; ++c) s4[c] = (T)0;
                    if (sl < nsl) {
                        const T *vj = SPILL && j == i ? vi : slot(j);
                        auto take = [&](int p, T *s) {
                            const auto x = ldp(vj + p * N), z = ldp(y + p * N);
#pragma unroll
                            for (int c = 0; c < N; ++c) s[c] += x.v[c] * z.v[c];
                        };
                        int p = sl * 8 + l8;
#pragma unroll (4 / H)
                        for (; p + (H - 1) * 8 * nsl < np; p += H * 8 * nsl) {
                            take(p, s4);
                            if constexpr (H == 2) take(p + 8 * nsl, s4 + N);
                        }
                        if (H == 2 && p < np) take(p, s4);
                    }
                    Sum<T> t;
                    if constexpr (H == 2) {
                        t.h = s4[0];
#pragma unroll
                        for (int c = 1; c < H * N; ++c) t.add(s4[c]);
                    } else t.h = s4[0] + s4[1];
                    t.fold(4);
                    t.fold(2);
                    t.fold(1);
                    const T a = t.rounded();
                    if (sl < nsl && l8 == 0) red[sl * nv + j] = a;
                };
                // ---- g = V^T v_i (v_i not scaled yet) while the halo arrives
                if (i > 0) {
                    dot(vi, s_red + KM);
                    for (int q = tid; q < nh; q += 2 * kWorkers) {
                        const int q2 = q + kWorkers, p = q < nhl ? q : q + nrow, p2 = q2 < nhl ? q2 : q2 + nrow;
                        const u64 *src = vb + (size_t)lo * B * WP;
                        unsigned v[2 * WP];
                        if constexpr (WP == 1) poll<2>(src + p, p2 - p, q2 < nh ? 2 : 1, tag - 1u, v, bound);
                        else {
                            unsigned a[2], b[2];
                            const int cnt = q2 < nh ? 2 : 1;
                            poll<2>(src + 2 * (size_t)p, 2 * (size_t)(p2 - p), cnt, tag - 1u, a, bound);
                            poll<2>(src + 2 * (size_t)p + 1, 2 * (size_t)(p2 - p), cnt, tag - 1u, b, bound);
                            v[0] = a[0];
                            v[1] = b[0];
                            v[2] = a[1];
                            v[3] = b[1];
                        }
                        halo[q] = from_words<T>(v);
                        if (q2 < nh) halo[q2] = from_words<T>(v + WP);
                    }
                    sync_workers();
                }
                // ---- w = M^-1 A v_i
                for (int q = tid; q < Rp; q += kWorkers) {
                    T y = (T)0;
                    if (q < nrow) {
                        const int u = k.u0 + q / B, r = q % B;
                        if (q < nc) {
#pragma unroll 4
                            for (int s = 0; s < W; ++s) {
                                T x[B], a[B];
                                load_x<B, T>(rv + ((size_t)s * nc + q) * B, a);
                                load_x<B, T>(X.template at<B>(ri[s * nc + q]), x);
                                y = row_add<B, T>(y, a, x);
                            }
                        } else y = row_times_x<B, T>(off, dc, ru, A, X, u, r);
                        const int id = B == 1 ? u : __ldg(nd + (size_t)u * B + r);
                        if (id == n) y = (T)0;
                        else if (pre == FG_PRECOND_DIAG) y *= __ldg(M + id);
                    }
                    w[q] = y;
                }
                sync_workers();
                if (B > 1 && pre == FG_PRECOND_BLOCKDIAG) {   // a node's rows are in this CTA
                    for (int q0 = 0; q0 < nrow; q0 += kWorkers / B * B) {
                        const int q = q0 + tid;
                        const bool on = tid < kWorkers / B * B && q < nrow;
                        T z = (T)0;
                        if (on) {
                            const int lu = q / B, u = k.u0 + lu;
                            if (__ldg(nd + (size_t)u * B + q % B) != n) {
                                T m[B];
                                load_vals<B, T>(M + ((size_t)u * B + q % B) * B, m);
                                z = m[0] * w[lu * B];
#pragma unroll
                                for (int c = 1; c < B; ++c) z += m[c] * w[lu * B + c];
                            }
                        }
                        sync_workers();
                        if (on) w[q] = z;
                    }
                    sync_workers();
                }
                // ---- s = V^T w over this CTA's rows; the first step's largest |w| in g's place
                dot(w, s_red);
                if (i == 0) {
                    T m = (T)0;
                    for (int q = tid; q < nrow; q += kWorkers) m = max(m, abs(w[q]));
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
                    if (lane == 0) s_red[KM + warp] = m;
                }
            }
            __syncthreads();                      // the Givens warp is done with column i - 2 too
            // ---- exchange: 2 nv sums (s_j, g_j), ||v_i||^2 and the stop flag
            if (tid < 2 * nv) {
                const int nsl = dot_slices(np, nv);
                const T *red = s_red + (tid & 1) * KM + (tid >> 1);
                T s = red[0];
                if (i == 0 && tid == 1)
                    for (int q = 1; q < kWorkers / 32; ++q) s = max(s, red[q]);
                else
                {
                    Sum<T> t;
                    for (int q = 0; q < nsl; ++q) t.add(red[q * nv]);
                    s = t.rounded();
                }
                if (g == 1) s_tot[tid] = s;
                else put<T>(part + ((size_t)tid * g + rank) * WP, s, tag);
            }
            // the norm: the Givens warp sums the warps' shares, then the CTAs'
            Sum<T> n2;
            if (!worker) {
                if (lane < kWorkers / 32) {
                    n2.h = s_n2h[lane];
                    if constexpr (sizeof(T) == 4) n2.l = s_n2l[lane];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) n2.fold(o);
                if (g > 1 && lane == 0) {
                    put_pair(norm + 2 * rank, n2, tag);
                    if (rank == 0) put1(note + (i & 1), (unsigned)s_stop, tag);
                }
            }
            if (g > 1 && worker) {
                if (direct) {
                    for (int m = gid; m < ((2 * nv + 3) & ~3); m += kGroups) {
                        Sum<T> t;
                        if (m < 2 * nv) {
                            const u64 *p = part + (size_t)m * g * WP;
                            if constexpr (WP == 1) {
                                unsigned v[kDirect32 / 8];
                                const int cnt = (g - l8 + 7) / 8;
                                poll<kDirect32 / 8>(p + l8, 8, cnt, tag, v, bound);
#pragma unroll
                                for (int q = 0; q < kDirect32 / 8; ++q) t.add(__uint_as_float(v[q]));
                            } else {
                                for (int q = l8; q < g; q += 8) {
                                    unsigned v[2];
                                    poll<2>(p + 2 * q, 1, 2, tag, v, bound);
                                    t.add(from_words<T>(v));
                                }
                            }
                        }
                        t.fold(4);
                        t.fold(2);
                        t.fold(1);
                        if (l8 == 0 && m < 2 * nv) s_tot[m] = t.rounded();
                    }
                } else {
                    // CTA `rank` sums slots rank, rank + g, ..., a warp each
                    for (int m = rank + warp * g; m < 2 * nv; m += g * (kWorkers / 32)) {
                        Sum<T> t;
                        const u64 *p = part + (size_t)m * g * WP;
                        constexpr int K = WP == 1 ? 10 : 5;
                        for (int q0 = lane; q0 < g; q0 += 32 * K) {
                            if constexpr (WP == 1) {
                                unsigned v[K];
                                poll<K>(p + q0, 32, (g - q0 + 31) / 32, tag, v, bound);
#pragma unroll
                                for (int q = 0; q < K; ++q) t.add(__uint_as_float(v[q]));
                            } else {
                                unsigned lo[K], hi[K];
                                poll<K>(p + 2 * q0, 64, (g - q0 + 31) / 32, tag, lo, bound);
                                poll<K>(p + 2 * q0 + 1, 64, (g - q0 + 31) / 32, tag, hi, bound);
#pragma unroll
                                for (int q = 0; q < K; ++q) {
                                    const unsigned v[2] = {lo[q], hi[q]};
                                    t.add(from_words<T>(v));
                                }
                            }
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) t.fold(o);
                        if (lane == 0) put<T>(total + m * WP, t.rounded(), tag);
                    }
                    if (tid < 2 * nv) {
                        unsigned v[WP];
                        poll<WP>(total + tid * WP, 1, WP, tag, v, bound);
                        s_tot[tid] = from_words<T>(v);
                    }
                }
            }
            if (!worker) {
                if (g > 1) {
                    Sum<T> t;
                    if (direct || rank == g - 1) {    // large gangs: CTA g - 1 sums it
                        constexpr int K = 5;
                        for (int q0 = lane; q0 < g; q0 += 32 * K) {
                            unsigned lw[K], hw[K];
                            poll<K>(norm + 2 * q0, 64, (g - q0 + 31) / 32, tag, lw, bound);
                            poll<K>(norm + 2 * q0 + 1, 64, (g - q0 + 31) / 32, tag, hw, bound);
#pragma unroll
                            for (int q = 0; q < K; ++q) {
                                const unsigned v[2] = {lw[q], hw[q]};
                                add_pair(t, v);
                            }
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) t.fold(o);
                        if (!direct && lane == 0) put_pair(total + (size_t)2 * km * WP, t, tag);
                    } else {
                        unsigned v[2];
                        poll<2>(total + (size_t)2 * km * WP, 1, 2, tag, v, bound);
                        add_pair(t, v);
                    }
                    n2 = t;
                }
                if (lane == 0) {
                    const T sc = i == 0 ? (T)1 : inv_norm(n2);     // v_0 is taken as it is
                    s_sc = sc;
                    if (i > 0) s_ss = sc * s_sg;
                    s_dg = gram_diag(n2, sc);
                }
            } else if (g > 1 && tid == kWorkers - 1 && rank != 0) {
                unsigned v[1];
                poll<1>(note + (i & 1), 0, 1, tag, v, bound);
                s_stop = (int)v[0];
            }
            if (__syncthreads_or(s_stop | s_gave_up)) break;   // (the flags may still change: one answer for all)
            const T sc = s_sc;
            T *c = s_c[i & 1];
            if (worker) {
                const T ss = i == 0 ? unit_scale(s_tot[1]) : s_ss;
                if (i == 0 && tid == 0) s_sg = ss;
                // ---- c = s - (G - I) s (times sg); the new Gram column from this step's sums
                for (int j = gid; j < ((nv + 3) & ~3); j += kGroups) {
                    T d = (T)0;
                    if (j < nv) {
                        const T gj = j == i ? s_dg : sc * s_tot[2 * j + 1];
                        for (int q = l8; q < nv; q += 8) {
                            const T e = q == i ? gj : j == i ? sc * s_tot[2 * q + 1] : E[j * km + q];
                            // V_i is unscaled in s_i too
                            d += e * (q == i ? sc * s_tot[2 * q] : s_tot[2 * q]);
                        }
                        if (l8 == 0) {
                            E[j * km + i] = gj;
                            if (j != i) E[i * km + j] = gj;
                        }
                    }
                    d += __shfl_xor_sync(0xffffffffu, d, 4);
                    d += __shfl_xor_sync(0xffffffffu, d, 2);
                    d += __shfl_xor_sync(0xffffffffu, d, 1);
                    if (l8 == 0 && j < nv) c[j] = ss * ((j == i ? sc * s_tot[2 * j] : s_tot[2 * j]) - d);
                }
                sync_workers();
                asm volatile("bar.arrive 2, %0;\n" ::"n"(kCycThreads) : "memory");
                // ---- v_i scaled, w scaled and times sg, w -= V c, ||w||^2; what neighbours need to vb
                // (FP32: four rows a thread, so that a coefficient is read once for
                // four; FP64: one, to keep every quarter of its pipe busy)
                Sum<T> t;
                const int keep_l = D.rw_hi * B, keep_r = nrow - D.rw_lo * B;
                constexpr int R = sizeof(T) == 4 ? 4 : 1;
                for (int q = tid * R; q < (SPILL ? Rp : nrow); q += kWorkers * R) {   // (SPILL: zeros behind the rows too)
                    T s0[R], s1[R], v[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        v[r] = sc * vi[q + r];
                        s0[r] = ss * w[q + r];
                        s1[r] = -c[i] * v[r];
                        (SPILL ? slot(i) : vi)[q + r] = v[r];
                    }
                    int j = 0;
                    const int in = SPILL ? min(i, js) : i;
#pragma unroll 4
                    for (; j + 1 < in; j += 2) {
                        const T c0 = c[j], c1 = c[j + 1];
                        T a[R], b[R];
                        if constexpr (R == 4) {
                            const auto x = ldp(V + (size_t)j * Rp + q), z = ldp(V + (size_t)(j + 1) * Rp + q);
#pragma unroll
                            for (int r = 0; r < R; ++r) { a[r] = x.v[r]; b[r] = z.v[r]; }
                        } else {
                            a[0] = V[(size_t)j * Rp + q];
                            b[0] = V[(size_t)(j + 1) * Rp + q];
                        }
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            s0[r] -= c0 * a[r];
                            s1[r] -= c1 * b[r];
                        }
                    }
                    if (j < in)
#pragma unroll
                        for (int r = 0; r < R; ++r) s0[r] -= c[j] * V[(size_t)j * Rp + q + r];
                    if constexpr (SPILL) {
                        for (int h = js; h < i; h += 8) {    // eight loads in flight
                            T a[8][R];
#pragma unroll
                            for (int m = 0; m < 8; ++m) {
                                const T *p = gV + (min(h + m, i - 1) - js) * gs + q;
                                if constexpr (R == 4) {
                                    const auto x = ldp(p);
#pragma unroll
                                    for (int r = 0; r < R; ++r) a[m][r] = x.v[r];
                                } else {
                                    a[m][0] = p[0];
                                }
                            }
#pragma unroll
                            for (int m = 0; m < 8; ++m) {
                                if (h + m >= i) break;
#pragma unroll
                                for (int r = 0; r < R; ++r) {
                                    if (m & 1) s1[r] -= c[h + m] * a[m][r];
                                    else s0[r] -= c[h + m] * a[m][r];
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        s0[r] += s1[r];
                        w[q + r] = s0[r];
                        if (g > 1 && q + r < nrow && (q + r < keep_l || q + r >= keep_r))
                            put<T>(vb + ((size_t)k.u0 * B + q + r) * WP, s0[r], tag);
                        t.add_square(s0[r]);
                    }
                }
                if (warp * 32 * R < nrow)
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t.fold(o);
                if (lane == 0) {
                    s_n2h[warp] = t.h;
                    if constexpr (sizeof(T) == 4) s_n2l[warp] = t.l;
                }
                sync_workers();                   // w complete (and the norm's shares)
            } else {
                // ---- the rotations of column i - 1 (H times s_sg), beside the rest of the step
                asm volatile("bar.sync 2, %0;\n" ::"n"(kCycThreads) : "memory");
                if (rank == 0 && i > 0) {
                    const bool stop = givens<T>(D.H, km, R, i - 1, s_c[(i - 1) & 1], 1.0 / (double)sc, target);
                    if (lane == 0) s_stop = stop;
                }
            }
        }
        __syncthreads();
        // ---- end of the cycle: y on rank 0, x += V y everywhere
        const unsigned ntag = base + (unsigned)km + 1u, ytag = ntag + 1u;
        double *y = s_t;
        if (!s_gave_up && !worker) {
            if (i == km - 1) {                    // the last vector's norm, for rank 0
                Sum<T> t;
                if (lane < kWorkers / 32) {
                    t.h = s_n2h[lane];
                    if constexpr (sizeof(T) == 4) t.l = s_n2l[lane];
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) t.fold(o);
                if (rank != 0) {
                    if (lane == 0) put_pair(norm2 + (i & 1) * (2 * (size_t)g) + 2 * rank, t, ntag);
                } else {
                    Sum<T> u;
                    if (lane == 0) u = t;
                    for (int q = lane; q < g; q += 32) {
                        if (q == 0) continue;
                        unsigned v[2];
                        poll<2>(norm2 + (i & 1) * (2 * (size_t)g) + 2 * q, 1, 2, ntag, v, bound);
                        add_pair(u, v);
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) u.fold(o);
                    __syncwarp();
                    if (!s_stop) givens<T>(D.H, km, R, i - 1, s_c[(i - 1) & 1], sqrt(u.value()), target);
                }
            }
            if (rank == 0) {
                const int m = R.steps;
                __syncwarp();
                back_substitute(D.H, km, s_g, m, y);
                for (int j = lane; j < m; j += 32) y[j] *= s_sg;
                if (g > 1)
                    for (int j = lane; j < m; j += 32) put<double>(note + 3 + 2 * j, y[j], ytag);
                if (lane == 0) {
                    if (g > 1) put1(note + 2, (unsigned)m, ytag);
                    s_m = m;
                }
            } else {
                unsigned v[1];
                poll<1>(note + 2, 0, 1, ytag, v, bound);
                for (int j = lane; j < (int)v[0] && j < km; j += 32) {
                    unsigned w2[2];
                    poll<2>(note + 3 + 2 * j, 1, 2, ytag, w2, bound);
                    y[j] = from_words<double>(w2);
                }
                if (lane == 0) s_m = min((int)v[0], km);
            }
            __syncwarp();
            if constexpr (sizeof(T) == 4) split_y(y, nullptr, s_m, s_tot, s_tot + 1, 2, s_a);
        }
        if (__syncthreads_or(s_gave_up)) {
            if (tid == 0) {
                atomicExch(&D.st->status, FG_ERR_TIMEOUT);
                D.st->live = D.st->in_cycle = 0;
            }
            return;
        }
        const int m = s_m;
        if (worker)
            for (int q = tid; q < nrow; q += kWorkers) {
                const int id = B == 1 ? k.u0 + q : __ldg(D.node_dof + (size_t)k.u0 * B + q);
                if (id == n) continue;
                Sum<T> t;
                for (int j = 0; j < m; ++j) {
                    const T v = slot(j)[q];
                    if constexpr (sizeof(T) == 8) t.h += y[j] * v;
                    else t.add_product(s_tot[2 * j], s_tot[2 * j + 1], v);
                }
                D.x[id] += sizeof(T) == 8 ? t.value() : t.value() * s_a[0];
            }
        if (rank == 0 && tid == kWorkers) {       // restart bookkeeping (pgmres.c:177-179)
            SysState *st = D.st;
            st->rho = R.rho;
            st->steps = m;
            st->iterations += R.iters;
            st->cycles += 1;
            st->in_cycle = 0;
            if (R.breakdown) { st->status = FG_ERR_BREAKDOWN; st->live = 0; }
            else if (!D.mixed) {
                if (!(st->rho > st->eps)) { st->converged = 1; st->live = 0; }
                else if (st->cycles >= D.lmax) { atomicCAS(&st->status, FG_OK, FG_ERR_NOTCONV); st->live = 0; }
            }
            *D.cy_epoch = base + (unsigned)km + 4u;
        }
    }
}

// dynamic shared memory of a gang CTA: the basis, the Gram matrix, the halo
size_t cycle_smem(int km, int rows, int halo_rows, size_t w)
{
    return w * ((size_t)km * rows + (((size_t)km * km + 3) & ~(size_t)3) + ((halo_rows + 3) & ~3));
}
template <typename T, bool SPILL> const void *cycle_kernel(int B)
{
    switch (B) {
    case 1: return (const void *)k_cycle<T, 1, SPILL>;
    case 2: return (const void *)k_cycle<T, 2, SPILL>;
    case 3: return (const void *)k_cycle<T, 3, SPILL>;
    default: return (const void *)k_cycle<T, 4, SPILL>;
    }
}
const void *cycle_kernel(int B, bool f64, bool spill)
{
    return f64 ? (spill ? cycle_kernel<double, true>(B) : cycle_kernel<double, false>(B))
               : (spill ? cycle_kernel<float, true>(B) : cycle_kernel<float, false>(B));
}

// What k_cycle<T, B> has on the current device: the dynamic shared memory with
// which one CTA fills an SM, and the CTAs that are then resident together (0:
// none).  Looked up once per device and kernel; raises the kernel's
// shared-memory limit there.
struct Residency { int ctas; size_t smem; };
Residency residency(int B, bool f64, bool spill = false)
{
    static std::mutex mu;
    static std::map<std::tuple<int, int, bool, bool>, Residency> found;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return {0, 0}; }
    std::lock_guard<std::mutex> l(mu);
    const auto key = std::make_tuple(dev, B, f64, spill);
    const auto it = found.find(key);
    if (it != found.end()) return it->second;
    Residency v{0, 0};
    const void *k = cycle_kernel(B, f64, spill);
    int coop = 0, occ = 0, sm = 0, own = 0;
    cudaFuncAttributes fa{};
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&own, cudaDevAttrReservedSharedMemoryPerBlock, dev) == cudaSuccess &&
        cudaFuncGetAttributes(&fa, k) == cudaSuccess && (size_t)sm > own + fa.sharedSizeBytes + 4096) {
        const size_t cap = ((size_t)sm - own - fa.sharedSizeBytes) & ~(size_t)127;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, kCycThreads, cap) == cudaSuccess && occ > 0)
            v = {sm_count(), cap};
    }
    cudaGetLastError();
    return found[key] = v;
}

}  // namespace

// CTAs of a system's gang: enough for its rows to fit shared memory, and,
// unless the batch is dense, while CTAs are left no more than gang_want rows
// each: below that a step is bound by the exchanges, whose words grow with the
// gang, above it by the rows (FP64: 52 FMA a row and step at kmax 30, two a
// cycle), so FP64 CTAs get rows as the square root of the units.  0: the system
// does not fit, or its numbering couples units too far apart for the halo.
// Measured with 512 / 256 / 128 rows FP32: 16k equations 4.70 / 4.32 / 4.46 ms a
// solve; with 128 / 96 / 64 rows FP64: 961 equations 2.02 / 1.99 / 1.89, a
// four-step process of 9k 19.1 / 17.0 / 18.2, 16k 5.62 / 5.69 / 5.69, Euler with
// 4k nodes 5.02 / 4.71 / 4.73; with 32 rows 961 equations 1.87, 9k 19.9.
// The halo needs no bound but its room: multi-dof meshes keep their node order, and
// with nodes numbered at random, where every CTA polls the whole newest vector, a step
// on chip / streaming takes FP64 (FP32) at 65 x 65 nodes of 2 dofs 17 / 32 us (13 / 29), of
// 3 25 / 35 (15 / 30), of 4 26 / 42 (16 / 36), at 129 x 129 of 2 FP32 25 / 35; larger ones
// have no room and stream.
static int gang_want(const fg_system *s, bool f64)
{
    return f64 ? std::max(64, (int)std::sqrt((double)s->topo.nunits)) : 256;
}
static int halo_units(const fg_system *s) { return std::min(s->topo.nunits, s->topo.rw_lo + s->topo.rw_hi); }
int gang_rows(const fg_system *s, int g);
int gang_size(const fg_system *s, int kmax, bool f64, bool dense)
{
    const int B = s->topo.ndof, nu = s->topo.nunits;
    const Residency dev = residency(B, f64);
    const int ctas = dev.ctas;
    if (ctas == 0 || nu == 0) return 0;
    const size_t w = f64 ? 8 : 4, fixed = cycle_smem(kmax, 0, halo_units(s) * B, w);
    if (fixed + (size_t)kmax * w * 64 > dev.smem || s->topo.rw_dc.empty()) return 0;   // (couplings that far fit no halo either)
    const int cap = (int)((dev.smem - fixed) / (kmax * w)) & ~3;
    const int cap_u = cap / B, want_u = dense ? cap_u : std::max(1, std::min(cap_u, gang_want(s, f64) / B));
    const int g = std::max((nu + cap_u - 1) / cap_u, std::min(ctas, (nu + want_u - 1) / want_u));
    return g <= ctas ? g : 0;
}
int set_gang_polls(long long polls)
{
    const int n = (int)std::min(polls, 0x7fffffffLL);
    FG_CUDA(cudaMemcpyToSymbol(g_gang_polls, &n, sizeof(n)));
    return FG_OK;
}
int gang_ctas(int B, bool f64, bool spill) { return residency(B, f64, spill).ctas; }
// Basis vectors that stay in shared memory when a system that does not fit
// runs alone on every CTA (0: fewer than a fifth, or none; it streams).
// Measured on FP64 systems (a step, streaming -> spilling): 147k equations,
// GMRES(30), 23 vectors inside 55 -> 34 us; 198k, GMRES(50), 12 inside 103 -> 65.
int gang_spill(const fg_system *s, int kmax, bool f64)
{
    const int B = s->topo.ndof;
    const Residency dev = residency(B, f64, true);
    if (dev.ctas == 0 || s->topo.nunits < dev.ctas || s->topo.rw_dc.empty()) return 0;
    const size_t w = f64 ? 8 : 4, fixed = cycle_smem(kmax, 0, halo_units(s) * B, w);
    if (fixed >= dev.smem) return 0;
    const int js = std::min(kmax - 2, (int)((dev.smem - fixed) / (w * gang_rows(s, dev.ctas))) - 2);
    return js >= 2 && 5 * js >= kmax ? js : 0;
}
int gang_rows(const fg_system *s, int g) { return ((s->topo.nunits + g - 1) / g * s->topo.ndof + 3) & ~3; }

// Exchange block of a gang: the epoch (16 bytes), the exchange words, the
// exchange vector.
static size_t gang_words(int kmax, int g, bool f64)
{
    const size_t w = f64 ? 2 : 1;
    return 4 * w * kmax * g + 4 * (size_t)g + 2 * w * kmax + 2 + 3 + 2 * (size_t)kmax;
}
static size_t gang_head(int kmax, int g, bool f64) { return 16 + (8 * gang_words(kmax, g, f64) + 15) / 16 * 16; }
size_t gang_bytes(const fg_system *s, int kmax, int g, bool f64)
{
    return gang_head(kmax, g, f64) + (size_t)s->topo.nunits * s->topo.ndof * (f64 ? 16 : 8);
}
size_t gang_spill_bytes(const fg_system *s, int kmax, int g, int js, bool f64)
{
    return js ? (size_t)(kmax - js) * g * gang_rows(s, g) * (f64 ? 8 : 4) : 0;
}
void set_gang_fields(SysDev &D, const fg_system *s, int kmax, int g, int js, bool f64)
{
    D.cy_js = js;
    D.cy_spill = s->ws.V.p;            // (free while the cycle is on chip)
    D.cy_g = g;
    if (!g) return;
    D.cy_rows = gang_rows(s, g);
    unsigned char *p = s->ws.gang.as<unsigned char>();
    D.cy_epoch = reinterpret_cast<unsigned *>(p);
    D.cy_part = reinterpret_cast<unsigned long long *>(p + 16);
    D.cy_vb = p + gang_head(kmax, g, f64);
}

// The CTAs of a cycle's launches: every rank of every live system (live empty:
// all) that has a gang, bin by bin, and the shared memory of a bin's largest.
void gang_items(const std::vector<SysDev> &hs, const std::vector<int> &live, int B, bool f64,
                std::vector<CycItem> &items, std::vector<CycBin> &bins)
{
    const size_t w = f64 ? 8 : 4;
    items.clear();
    bins.clear();
    int nbin = 0;
    for (const SysDev &D : hs) nbin = std::max(nbin, D.cy_bin + 1);
    for (int b = 0; b < nbin; ++b) {
        CycBin bin{(int)items.size(), 0, 0, false};
        for (int i = 0; i < (int)hs.size(); ++i) {
            const SysDev &D = hs[i];
            if (D.cy_g == 0 || D.cy_bin != b || (!live.empty() && !live[i])) continue;
            for (int r = 0; r < D.cy_g; ++r)
                items.push_back({i, r, (int)((long long)D.nunits * r / D.cy_g), (int)((long long)D.nunits * (r + 1) / D.cy_g)});
            // and the operator's rows, as far as they fit
            const size_t cap = residency(B, f64, D.cy_js > 0).smem;
            const size_t need = cycle_smem(D.kmax, 0, 0, w) + w * (D.cy_js > 0 ? D.cy_js + 2 : D.kmax) * D.cy_rows +
                                cycle_smem(0, 0, std::min(D.nunits, D.rw_lo + D.rw_hi) * B, w);
            bin.smem = std::max(bin.smem, std::min(cap, need + (size_t)D.cy_rows * D.rw_w * (B * w + 2) + 16));
            bin.spill = bin.spill || D.cy_js > 0;
        }
        bin.ctas = (int)items.size() - bin.first;
        if (bin.ctas) bins.push_back(bin);
    }
}

int launch_cycle(int B, bool f64, bool spill, const SysDev *sys, const CycItem *items, int ctas, size_t smem,
                 cudaStream_t st)
{
    int bytes = (int)smem;
    void *args[] = {(void *)&sys, (void *)&items, (void *)&bytes};
    const void *k = cycle_kernel(B, f64, spill);
    cudaError_t e = cudaLaunchCooperativeKernel(k, dim3(ctas), dim3(kCycThreads), args, smem, st);
    if (e != cudaSuccess) cuda_fail(e, "cudaLaunchCooperativeKernel");
    return 1;
}

}  // namespace fg
