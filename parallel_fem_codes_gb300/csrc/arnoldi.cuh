// Arnoldi step and cycle-end kernels of the streaming restart cycle
// (included by krylov.cu): two passes over the basis per step, V read once in
// each.
//
// The basis is kept unscaled: V[j] is the vector as the step left it and
// vscale[j] the reciprocal of its norm, known when the step's last part sums
// it, so that no pass is spent on scaling (an FP16 basis is scaled when it is
// stored, vscale[j] = 1 / sigma).  A step leaves its vector times vscale[kmax], a
// power of two that the cycle's first step finds (unit_scale).  Both passes walk parts of kPartMin..kPartMax
// dofs (the size is chosen per batch from its total dofs), a 16-byte pack of
// every vector per thread and several basis vectors in flight.  A part is one
// CTA's, or, where a batch has few parts, gridDim.y CTAs': pass 1 splits the
// basis vectors among them, pass 2 the dofs.  Part results are combined by the last part of the system in fixed
// order.  HBM-bound in FP32; in FP64 the FP64 pipe (2 FMA per clock and SM)
// binds: 3 (i + 1) FMA per dof and step.

// 16-byte packs along the dof direction: parts start at multiples of the
// pack width and vectors are zero beyond n up to n_pad, so a pack never
// straddles two parts and reads past n see zeros.
template <typename T> struct Pk {
    static constexpr int N = 16 / sizeof(T);
    struct alignas(16) type { T v[N]; };
};
template <typename T> __device__ __forceinline__ typename Pk<T>::type ld_pk(const T *p)
{
    return *reinterpret_cast<const typename Pk<T>::type *>(p);
}
template <typename T> __device__ __forceinline__ void st_pk(T *p, const typename Pk<T>::type &v)
{
    *reinterpret_cast<typename Pk<T>::type *>(p) = v;
}

// The basis may be stored in a narrower type TV than the arithmetic type T
// (FP16 under FP32 arithmetic): a basis pack is 16 bytes of TV, G dofs; the
// work vectors are read and written G dofs at a time as G / Pk<T>::N packs.
template <typename TV> struct VPk { static constexpr int G = 16 / sizeof(TV); };

template <typename T, int G> __device__ __forceinline__ void ld_g(const T *p, T (&o)[G])
{
    constexpr int N = Pk<T>::N;
#pragma unroll
    for (int h = 0; h < G / N; ++h) {
        const auto v = ld_pk(p + h * N);
#pragma unroll
        for (int c = 0; c < N; ++c) o[h * N + c] = v.v[c];
    }
}
template <typename T, int G> __device__ __forceinline__ void st_g(T *p, const T (&o)[G])
{
    constexpr int N = Pk<T>::N;
#pragma unroll
    for (int h = 0; h < G / N; ++h) {
        typename Pk<T>::type v;
#pragma unroll
        for (int c = 0; c < N; ++c) v.v[c] = o[h * N + c];
        st_pk(p + h * N, v);
    }
}
// 16 bytes of the basis, which passes through: L1 is left to the vectors that
// every group of basis vectors reads again
__device__ __forceinline__ uint4 ld_stream(const void *p)
{
    uint4 r;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
// one basis pack as T (KEEP: read again soon)
template <typename T, typename TV, bool KEEP = false>
__device__ __forceinline__ void ld_v(const TV *p, T (&o)[VPk<TV>::G])
{
    if constexpr (std::is_same<TV, __half>::value) {
        const uint4 r = KEEP ? *reinterpret_cast<const uint4 *>(p) : ld_stream(p);
        const unsigned u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            __half2 hv;
            memcpy(&hv, &u[h], 4);
            const float2 f = __half22float2(hv);
            o[2 * h] = (T)f.x;
            o[2 * h + 1] = (T)f.y;
        }
    } else {
        const uint4 r = KEEP ? *reinterpret_cast<const uint4 *>(p) : ld_stream(p);
        memcpy(&o[0], &r, 16);
    }
}
template <typename T, typename TV>
__device__ __forceinline__ void st_v(TV *p, const T (&o)[VPk<TV>::G])
{
    if constexpr (std::is_same<TV, __half>::value) {
        unsigned u[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const __half2 hv = __floats2half2_rn((float)o[2 * h], (float)o[2 * h + 1]);
            memcpy(&u[h], &hv, 4);
        }
        *reinterpret_cast<uint4 *>(p) = make_uint4(u[0], u[1], u[2], u[3]);
    } else {
        st_g<T, VPk<TV>::G>(reinterpret_cast<T *>(p), o);
    }
}

constexpr int kMaxSplit = 8;        // CTAs of a part in pass 2

// <V[j], w> and <V[j], V[i]> over a part for this CTA's share of j = 0..i, raw
// (V and w as stored).  A thread holds a pack of w and of V[i] and JB basis vectors' packs
// at a time, so that JB + 2 loads are in flight and w is read from L1 after
// the first group; the 2 JB sums are folded over the warp by halving (a
// value's lanes drop out as the values do), then over the warps (FP32: in
// pairs).
template <typename T, typename TV>
__device__ __forceinline__ void part_dots(const SysDev &D, const DChunk &k, int i, const T *__restrict__ w, T (*sw)[2 * kMaxRestart],
                                          double *out)
{
    constexpr int G = VPk<TV>::G, JB = sizeof(T) == 8 ? 4 : sizeof(TV) == 2 ? 4 : 8, NV = 2 * JB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nv = i + 1;
    const TV *V = (const TV *)D.V;
    const size_t ld = (size_t)D.n_pad;
    const TV *vi = V + (size_t)i * ld;
    const int ng = (nv + JB - 1) / JB;
    const int ja = JB * (int)(ng * blockIdx.y / gridDim.y), jb = min(nv, JB * (int)(ng * (blockIdx.y + 1) / gridDim.y));
    for (int j0 = ja; j0 < jb; j0 += JB) {
        T s[NV];
#pragma unroll
        for (int u = 0; u < NV; ++u) s[u] = (T)0;
        for (int q = k.d0 + threadIdx.x * G; q < k.d1; q += kThreads * G) {
            T w0[G], u0[G], v[JB][G];
#pragma unroll
            for (int u = 0; u < JB; ++u)
                if (j0 + u <= i) ld_v<T, TV>(V + (j0 + u) * ld + q, v[u]);
                else
#pragma unroll
                    for (int c = 0; c < G; ++c) v[u][c] = (T)0;
            ld_g<T, G>(w + q, w0);
            ld_v<T, TV, true>(vi + q, u0);
#pragma unroll
            for (int u = 0; u < JB; ++u)
#pragma unroll
                for (int c = 0; c < G; ++c) {
                    s[u] += v[u][c] * w0[c];
                    s[JB + u] += v[u][c] * u0[c];
                }
        }
        Sum<T> t[NV];
#pragma unroll
        for (int u = 0; u < NV; ++u) t[u].h = s[u];
        int o = 16;
#pragma unroll
        for (int m = NV / 2; m >= 1; m >>= 1, o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int u = 0; u < m; ++u) {
                const Sum<T> give = up ? t[u] : t[u + m];
                if (up) t[u] = t[u + m];
                t[u].take(give, o);
            }
        }
        for (; o > 0; o >>= 1) t[0].fold(o);
        // value index: the lane's upper bits, most significant first
        constexpr int SH = NV == 16 ? 1 : 2;
        const int idx = lane >> SH, j = j0 + (idx & (JB - 1));
        if ((lane & ((1 << SH) - 1)) == 0 && j < nv) sw[warp][(idx < JB ? 0 : nv) + j] = t[0].rounded();
    }
    __syncthreads();
    for (int h = threadIdx.x; h < 2 * (jb - ja); h += kThreads) {
        const int j = h < jb - ja ? ja + h : nv + ja + h - (jb - ja);
        Sum<T> t;
#pragma unroll
        for (int q = 0; q < kThreads / 32; ++q) t.add(sw[q][j]);
        out[j] = t.value();
    }
}

// Pass 1 (classical Gram-Schmidt with a Gram correction): s = V^T w (w = M^-1 A
// v_i from the matvec) and the new column g = V^T v_i of the basis' Gram
// matrix G in one sweep.  The last part forms c = s + (s - G s): the
// coefficients of the two classical passes of CGS2 (h1 = s, h2 = V^T (w - V s) =
// s - G s, but for rounding) with the second one taken from G instead of a second sweep; c becomes
// column i of H and, unscaled, the update that k_orth applies, the scale of w behind it.
template <typename T, typename TV>
__global__ void __launch_bounds__(kThreads, 3)
k_dots(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch, int i)
{
    __shared__ T sw[kThreads / 32][2 * kMaxRestart], mx[kThreads / 32];
    __shared__ double tot[2 * kMaxRestart];
    constexpr bool kUnscaled = std::is_same<T, TV>::value;
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->in_cycle) continue;
        __syncthreads();
        part_dots<T, TV>(D, k, i, (const T *)D.w, sw, D.part + k.part * kPartStride);
        if (kUnscaled && i == 0) {               // the part's largest |w| (one CTA a part here)
            constexpr int G = VPk<TV>::G;
            T m = (T)0;
            for (int q = k.d0 + threadIdx.x * G; q < k.d1; q += kThreads * G) {
                T v[G];
                ld_g<T, G>((const T *)D.w + q, v);
#pragma unroll
                for (int e = 0; e < G; ++e) m = max(m, abs(v[e]));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if ((threadIdx.x & 31) == 0) mx[threadIdx.x >> 5] = m;
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int q = 1; q < kThreads / 32; ++q) m = max(m, mx[q]);
                D.part[k.part * kPartStride + 2] = (double)m;
            }
        }
        if (last_part(D, 1, gridDim.y)) {
            reduce_parts(D, 2 * (i + 1) + (kUnscaled && i == 0), tot);
            const int km = D.kmax;
            const double *vs = D.vscale;
            const double ws = kUnscaled ? vs[i] : 1.0;   // the scale of w as stored
            if (i == 0 && threadIdx.x == 0) D.vscale[km] = kUnscaled ? (double)unit_scale((T)tot[2]) : 1.0;
            for (int j = threadIdx.x; j <= i; j += kThreads) {
                const double g = tot[i + 1 + j] * vs[j] * vs[i];
                D.G[j * km + i] = g;
                D.G[i * km + j] = g;
                tot[j] *= vs[j] * ws;
            }
            __syncthreads();
            if (threadIdx.x == 0) D.hbuf[i + 1] = ws * vs[km];
            for (int j = threadIdx.x; j <= i; j += kThreads) {
                double gs = 0.0;
                for (int l = 0; l <= i; ++l) gs += D.G[l * km + j] * tot[l];
                const double cj = tot[j] + (tot[j] - gs);
                D.hcol[j] = cj;
                D.hbuf[j] = cj * vs[j] * vs[km];
            }
        }
    }
}

// Pass 2: the new vector w - V c, unscaled, into V[i+1] (an FP16 basis: in
// place, k_normalize stores it), and its norm; then, in the last part, the
// Givens step and the cycle's stop test.
template <typename T, typename TV>
__global__ void __launch_bounds__(kThreads, 3)
k_orth(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch, int i)
{
    constexpr int G = VPk<TV>::G, JB = sizeof(TV) == 2 ? 4 : 8;
    __shared__ T hs[kMaxRestart + 4];
    __shared__ double red[kThreads / 32], st_t[kMaxRestart + 4], st_a[kMaxRestart + 4], tot[kMaxSplit];
    const int total = *nch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[total - 1 - c];      // pass 1's last parts first: those are in L2
        const SysDev &D = sys[k.sys];
        if (!D.st->in_cycle) continue;
        __syncthreads();
        for (int j = threadIdx.x; j <= i + 1; j += kThreads) hs[j] = (T)D.hbuf[j];
        __syncthreads();
        const TV *V = (const TV *)D.V;
        const size_t ld = (size_t)D.n_pad;
        const T *w = (const T *)D.w;
        T *out = std::is_same<T, TV>::value ? (T *)D.V + (size_t)(i + 1) * ld : (T *)D.w;
        const T ws = hs[i + 1];
        Sum<T> nrm;
        const int len = k.d1 - k.d0;
        const int d0 = k.d0 + ((int)((long long)len * blockIdx.y / gridDim.y) & ~7);
        const int d1 = blockIdx.y + 1 == gridDim.y ? k.d1 : k.d0 + ((int)((long long)len * (blockIdx.y + 1) / gridDim.y) & ~7);
        for (int q = d0 + threadIdx.x * G; q < d1; q += kThreads * G) {
            T s0[G], s1[G];
            ld_g<T, G>(w + q, s0);
#pragma unroll
            for (int u = 0; u < G; ++u) { s0[u] *= ws; s1[u] = (T)0; }
            int j = 0;
            for (; j + JB <= i + 1; j += JB) {
                T v[JB][G];
#pragma unroll
                for (int u = 0; u < JB; ++u) ld_v<T, TV>(V + (j + u) * ld + q, v[u]);
#pragma unroll
                for (int u = 0; u < JB; u += 2) {
                    const T h0 = hs[j + u], h1 = hs[j + u + 1];
#pragma unroll
                    for (int e = 0; e < G; ++e) {
                        s0[e] -= h0 * v[u][e];
                        s1[e] -= h1 * v[u + 1][e];
                    }
                }
            }
            if (j <= i) {                     // the rest
                T v[JB][G];
#pragma unroll
                for (int u = 0; u < JB - 1; ++u)
                    if (j + u <= i) ld_v<T, TV>(V + (j + u) * ld + q, v[u]);
#pragma unroll
                for (int u = 0; u < JB - 1; ++u) {
                    if (j + u > i) break;
                    const T h0 = hs[j + u];
#pragma unroll
                    for (int e = 0; e < G; ++e) s0[e] -= h0 * v[u][e];
                }
            }
#pragma unroll
            for (int e = 0; e < G; ++e) {
                s0[e] = q + e < D.n ? s0[e] + s1[e] : (T)0;
                nrm.add_square(s0[e]);
            }
            st_g<T, G>(out + q, s0);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm.fold(o);
        if (lane == 0) red[warp] = nrm.value();
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0;
            for (int w8 = 0; w8 < kThreads / 32; ++w8) s += red[w8];
            D.part[k.part * kPartStride + blockIdx.y] = s;
        }
        if (last_part(D, 3, gridDim.y)) {
            reduce_parts(D, gridDim.y, tot);
            if (warp == 0) {
                SysState *st = D.st;
                double n2 = tot[0];
                for (int y = 1; y < gridDim.y; ++y) n2 += tot[y];
                const double vn = sqrt(n2), hn = vn / D.vscale[D.kmax];
                Rot R{D.cs, D.sn, D.g, st_t, st_a, 0, 0, 0, 0.0};
                const bool stop = givens<double>(D.H, D.kmax, R, i, D.hcol, hn, D.mixed ? st->target : st->eps);
                __syncwarp();
                if (lane == 0) {
                    st->hn = hn;
                    D.vscale[i + 1] = std::is_same<T, TV>::value ? 1.0 / vn : (double)D.vsci;
                    st->rho = R.rho;
                    st->steps = R.steps;
                    st->iterations += 1;
                    if (R.breakdown) st->status = FG_ERR_BREAKDOWN;
                    if (stop) st->in_cycle = 0;
                }
                if (stop) back_substitute(D.H, D.kmax, D.g, R.steps, D.y);
            }
        }
    }
}

// FP16 basis: v_{i+1} = w * (1 / h_{i+1,i}) (pgmres.c:117), stored as sigma v
template <typename T, typename TV>
__global__ void __launch_bounds__(kThreads)
k_normalize(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch, int i)
{
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->in_cycle) continue;
        const T sc = (T)((double)D.vsc / D.st->hn);
        const T *w = (const T *)D.w;
        TV *v = (TV *)D.V + (size_t)(i + 1) * D.n_pad;
        constexpr int G = VPk<TV>::G;
        for (int q = k.d0 + threadIdx.x * G; q < k.d1; q += kThreads * G) {
            T p[G];
            ld_g<T, G>(w + q, p);
#pragma unroll
            for (int c = 0; c < G; ++c) p[c] = q + c < D.n ? sc * p[c] : (T)0;
            st_v<T, TV>(v + q, p);
        }
    }
}

// ---------------------------------------------------------------- cycle end
// x += V y (pgmres.c:173-175) with y from k_orth; the last part does the
// restart bookkeeping (:177-179).  FP32: the sum of the products in FP32 pairs (split_y).
template <typename T, typename TV>
__global__ void __launch_bounds__(kThreads)
k_update(const SysDev *__restrict__ sys, const DChunk *__restrict__ ch, const int *__restrict__ nch)
{
    __shared__ double y[kMaxRestart], back;
    __shared__ float yh[kMaxRestart], yl[kMaxRestart];
    const int total = *nch;
    for (int c = blockIdx.x; c < total; c += gridDim.x) {
        const DChunk k = ch[c];
        const SysDev &D = sys[k.sys];
        if (!D.st->live) continue;
        const int m = D.st->steps;
        __syncthreads();
        if constexpr (sizeof(T) == 8) {
            for (int j = threadIdx.x; j < m; j += kThreads) y[j] = D.y[j] * D.vscale[j];
        } else if (threadIdx.x < 32) split_y(D.y, D.vscale, m, yh, yl, 1, &back);
        __syncthreads();
        const TV *V = (const TV *)D.V;
        const size_t ld = (size_t)D.n_pad;
        // (x and V are zero-padded to n_pad, so the pack past n adds zeros)
        constexpr int N = VPk<TV>::G;
        for (int q = k.d0 + threadIdx.x * N; q < k.d1; q += kThreads * N) {
            Sum<T> s[N];
            auto take = [&](int j, const T (&v)[N]) {
#pragma unroll
                for (int e = 0; e < N; ++e) {
                    if constexpr (sizeof(T) == 8) s[e].h += v[e] * y[j];
                    else s[e].add_product(yh[j], yl[j], v[e]);
                }
            };
            int j = 0;
            for (; j + 3 < m; j += 4) {
                T v0[N], v1[N], v2[N], v3[N];
                ld_v<T, TV>(V + j * ld + q, v0);
                ld_v<T, TV>(V + (j + 1) * ld + q, v1);
                ld_v<T, TV>(V + (j + 2) * ld + q, v2);
                ld_v<T, TV>(V + (j + 3) * ld + q, v3);
                take(j, v0);
                take(j + 1, v1);
                take(j + 2, v2);
                take(j + 3, v3);
            }
            for (; j < m; ++j) {
                T v0[N];
                ld_v<T, TV>(V + j * ld + q, v0);
                take(j, v0);
            }
#pragma unroll
            for (int e = 0; e < N; e += 2) {
                double2 x2 = *reinterpret_cast<const double2 *>(D.x + q + e);
                x2.x += sizeof(T) == 8 ? s[e].value() : s[e].value() * back;
                x2.y += sizeof(T) == 8 ? s[e + 1].value() : s[e + 1].value() * back;
                *reinterpret_cast<double2 *>(D.x + q + e) = x2;
            }
        }
        if (last_part(D, 4)) {
            if (threadIdx.x == 0) {
                SysState *st = D.st;
                st->cycles += 1;
                st->in_cycle = 0;
                if (st->status == FG_ERR_BREAKDOWN) { st->live = 0; }
                else if (!D.mixed) {
                    if (!(st->rho > st->eps)) { st->converged = 1; st->live = 0; }
                    else if (st->cycles >= D.lmax) { st->status = FG_ERR_NOTCONV; st->live = 0; }
                }
            }
        }
    }
}
