// kernels.cuh -- sm_100a kernels of the RSFE Split-Bregman path, templated on the
// arithmetic type T (float or double).
//
// Reference routines restated here (paths relative to the reference project):
//   Gaussian filter      header/convolution_imp.hxx:22-91, :535-653
//   Heaviside            header/rsfe_splitbregman_imp.hxx:174-192
//   fitting terms + rhs  header/rsfe_splitbregman_imp.hxx:1700-1761
//   Gauss-Seidel         header/poisson_imp.hxx:23-336 (Neumann), :340-429 (Dirichlet)
//   clamp, tolerance     header/rsfe_splitbregman_imp.hxx:320-339, :1832
//   grad, div            header/image3d_imp.hxx:744-889, :948-1384
//   shrink, Bregman      header/rsfe_splitbregman_imp.hxx:343-365, :1868-1932
//   edge detector        header/rsfe_splitbregman_imp.hxx:196-316 (GRAD branch)
#pragma once

#include <type_traits>

#include "common.cuh"

namespace im3d {

constexpr int NH_MAX = 129;  // largest Gaussian support handled by the conv kernels

// ------------------------------------------------------------------ Heaviside
// H(x) = 1/2 (1 + 2/pi atan(x/eps)) and 1 - H(x) = H(-x), both to full relative
// precision: the smaller of the two is atan(1/|y|)/pi for |y| >= 1 (no cancellation
// against 1/2), the larger is 1 minus it. With eps = 1e-3 the smaller value reaches
// ~3e-4 and the fitting terms divide by its convolution, so FP32 needs this form.
template <typename T>
__device__ __forceinline__ void heaviside_pair(T phi, T center, T inv_eps, T& H, T& Hb)
{
    const T inv_pi = T(0.318309886183790671537767526745028724);
    const T x = (phi - center) * inv_eps;
    const T y = fabs(x);
    // one arctangent, of 1/y or y, and selects instead of branches
    const bool big = y >= T(1);
    T arg = y;
    if (big) {
        if constexpr (sizeof(T) == 4) arg = __frcp_rn(y);  // = 1.0f / y, correctly rounded
        else arg = T(1) / y;
    }
    const T at = atan(arg);
    const T small = big ? at * inv_pi : T(0.5) - at * inv_pi;
    const T large = T(1) - small;
    if (x > T(0)) { H = large; Hb = small; }
    else { H = small; Hb = large; }
}

// ------------------------------------------------------------ loaders/storers
// A loader's raw() issues the memory reads of one cell and cook() turns them into the
// staged fields, so that a pass can issue the reads of all its cells before it
// computes any of them; operator() does both.
template <typename T, int N>
struct LdVec {
    const Vec<T, N>* p;
    Dims d;
    typedef Vec<T, N> Raw;
    __device__ __forceinline__ Raw raw(int i, int j, int k) const { return p[d.idx(i, j, k)]; }
    __device__ __forceinline__ Vec<T, N> cook(const Raw& r) const { return r; }
    __device__ __forceinline__ Vec<T, N> operator()(int i, int j, int k) const
    {
        return p[d.idx(i, j, k)];
    }
};

// A storer's pre() issues the reads that its store of cells k0 .. k0+cnt-1 of one row
// needs, early in a pass, and put4() stores those cells; operator() stores one cell.
template <typename T, int N>
struct StVec {
    Vec<T, N>* p;
    Dims d;
    struct Pre {};
    __device__ __forceinline__ Pre pre(int, int, int, int) const { return Pre{}; }
    __device__ __forceinline__ void put4(const Pre&, int i, int j, int k0, const Vec<T, N> (&v)[4],
                                         int cnt) const
    {
        const long long q = d.idx(i, j, k0);
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r < cnt) p[q + r] = v[r];
    }
    __device__ __forceinline__ void operator()(int i, int j, int k, const Vec<T, N>& v) const
    {
        p[d.idx(i, j, k)] = v;
    }
};

template <typename T>
struct LdScalar {
    const T* p;
    Dims d;
    typedef Vec<T, 1> Raw;
    __device__ __forceinline__ Raw raw(int i, int j, int k) const { return (*this)(i, j, k); }
    __device__ __forceinline__ Vec<T, 1> cook(const Raw& r) const { return r; }
    __device__ __forceinline__ Vec<T, 1> operator()(int i, int j, int k) const
    {
        Vec<T, 1> r;
        r.v[0] = ld_g(p + d.idx(i, j, k));
        return r;
    }
};

template <typename T>
struct LdOne {
    typedef Vec<T, 1> Raw;
    __device__ __forceinline__ Raw raw(int i, int j, int k) const { return (*this)(i, j, k); }
    __device__ __forceinline__ Vec<T, 1> cook(const Raw& r) const { return r; }
    __device__ __forceinline__ Vec<T, 1> operator()(int, int, int) const
    {
        Vec<T, 1> r;
        r.v[0] = T(1);
        return r;
    }
};

template <typename T>
struct StScalar {
    T* p;
    Dims d;
    struct Pre {};
    __device__ __forceinline__ Pre pre(int, int, int, int) const { return Pre{}; }
    __device__ __forceinline__ void put4(const Pre&, int i, int j, int k0, const Vec<T, 1> (&v)[4],
                                         int cnt) const
    {
        const long long q = d.idx(i, j, k0);
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r < cnt) p[q + r] = v[r].v[0];
    }
    __device__ __forceinline__ void operator()(int i, int j, int k, const Vec<T, 1>& v) const
    {
        p[d.idx(i, j, k)] = v.v[0];
    }
};

// four consecutive values from p (16-byte vector reads when they are aligned), zero
// past cnt
template <typename T>
__device__ __forceinline__ void ld4(const T* __restrict__ p, int cnt, T (&o)[4])
{
    if (cnt == 4 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
        if constexpr (sizeof(T) == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(p));
            o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
        } else {
            const double2 a = __ldg(reinterpret_cast<const double2*>(p));
            const double2 b = __ldg(reinterpret_cast<const double2*>(p) + 1);
            o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
        }
    } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) o[r] = r < cnt ? ld_g(p + r) : T(0);
    }
}

// two values to p and p+1: one vector store when aligned
template <typename T>
__device__ __forceinline__ void st2(T* p, T a, T b)
{
    if ((reinterpret_cast<uintptr_t>(p) & (2 * sizeof(T) - 1)) == 0) {
        Vec<T, 2> v;
        v.v[0] = a;
        v.v[1] = b;
        *reinterpret_cast<Vec<T, 2>*>(p) = v;
    } else {
        p[0] = a;
        p[1] = b;
    }
}

// Stage-1 input: (H u0, H, Hb u0, Hb) from phi and u0.
template <typename T>
struct LdHeaviside {
    const T* phi;
    const T* u0;
    Dims d;
    T center, inv_eps;
    struct Raw {
        T phi, u;
    };
    __device__ __forceinline__ Raw raw(int i, int j, int k) const
    {
        const long long q = d.idx(i, j, k);
        return Raw{ld_g(phi + q), ld_g(u0 + q)};
    }
    __device__ __forceinline__ Vec<T, 4> cook(const Raw& w) const
    {
        T H, Hb;
        heaviside_pair(w.phi, center, inv_eps, H, Hb);
        Vec<T, 4> r;
        r.v[0] = H * w.u;
        r.v[1] = H;
        r.v[2] = Hb * w.u;
        r.v[3] = Hb;
        return r;
    }
    __device__ __forceinline__ Vec<T, 4> operator()(int i, int j, int k) const { return cook(raw(i, j, k)); }
};

// Forcing term of the Poisson step (rsfe_splitbregman_imp.hxx:1750-1761), from
// (kr2, kr1) = K * (l1 f1 - l2 f2, l1 f1^2 - l2 f2^2), in the reference's order:
//   r = kr2*u0*2 - (l1-l2)*u0*u0*kones - kr1, r /= lamda, r -= divdb.
// mode 0: natural rhs. mode 1: colour-packed rhs and colour-packed copy of phi.
// mode 2: colour-packed b_eff = rhs + phi/dt, packed phi, and sum b_eff^2.
// Dirichlet: the packed phi takes the boundary value on the faces.
template <typename T>
struct StRhs {
    const T* u0;
    const T* kones;  // NULL when lamda1 == lamda2 (the term is exactly zero)
    const T* divdb;
    const T* phi;
    T* out;      // natural rhs (mode 0) or packed rhs / b_eff (modes 1, 2)
    T* upk;      // packed phi (modes 1, 2)
    double* beff2;
    Dims d;
    T l12, lamda, inv_dt, bc;
    T inv_lamda;  // FP32 multiplies by it instead of dividing (same value when lamda is a power of two)
    int mode, dirichlet;
    struct Pre {
        T u[4], kn[4], dv[4], ph[4];
    };
    __device__ __forceinline__ Pre pre(int i, int j, int k0, int cnt) const
    {
        Pre w;
        const long long q = d.idx(i, j, k0);
        ld4(u0 + q, cnt, w.u);
        if (kones) ld4(kones + q, cnt, w.kn);
        ld4(divdb + q, cnt, w.dv);
        if (mode != 0) ld4(phi + q, cnt, w.ph);
        return w;
    }
    // the forcing term of one cell, operations as in operator()
    __device__ __forceinline__ T force(const Pre& w, int r, const Vec<T, 2>& v) const
    {
        const T u = w.u[r];
        T f = v.v[0];
        f *= u;
        f *= T(2);
        if (kones) {
            T a = l12;
            a *= u;
            a *= u;
            a *= w.kn[r];
            f -= a;
        }
        f -= v.v[1];
        if constexpr (sizeof(T) == 4) f *= inv_lamda;
        else f /= lamda;
        f -= w.dv[r];
        return f;
    }
    // k0 is even: cells k0, k0+2 have the colour of k0 and packed slots k0/2, k0/2+1,
    // cells k0+1, k0+3 the other colour and the same two slots
    __device__ __forceinline__ void put4(const Pre& w, int i, int j, int k0, const Vec<T, 2> (&v)[4],
                                         int cnt) const
    {
        T f[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) f[r] = force(w, r, v[r]);
        if (mode == 0) {
            T* o = out + d.idx(i, j, k0);
            if (cnt == 4) {
                st2(o, f[0], f[1]);
                st2(o + 2, f[2], f[3]);
            } else {
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < cnt) o[r] = f[r];
            }
            return;
        }
        const bool face_ij = i == 0 || j == 0 || i == d.nx - 1 || j == d.ny - 1;
        T ph[4], val[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            ph[r] = w.ph[r];
            if (dirichlet && (face_ij || k0 + r == 0 || k0 + r == d.nz - 1)) ph[r] = bc;
            val[r] = mode == 2 ? f[r] + ph[r] * inv_dt : f[r];
        }
        const int c0 = (i + j + k0) & 1;
        const long long base = d.pidx(i, j, k0);
        const long long o0 = base + (c0 ? d.npk() : 0), o1 = base + (c0 ? 0 : d.npk());
        if (cnt == 4) {
            st2(upk + o0, ph[0], ph[2]);
            st2(upk + o1, ph[1], ph[3]);
            st2(out + o0, val[0], val[2]);
            st2(out + o1, val[1], val[3]);
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (r < cnt) {
                    const long long o = ((r & 1) ? o1 : o0) + (r >> 1);
                    upk[o] = ph[r];
                    out[o] = val[r];
                }
            }
        }
    }
    __device__ __forceinline__ void operator()(int i, int j, int k, const Vec<T, 2>& v) const
    {
        const long long q = d.idx(i, j, k);
        const T u = ld_g(u0 + q);
        T r = v.v[0];
        r *= u;
        r *= T(2);
        if (kones) {
            T a = l12;
            a *= u;
            a *= u;
            a *= ld_g(kones + q);
            r -= a;
        }
        r -= v.v[1];
        if constexpr (sizeof(T) == 4) r *= inv_lamda;
        else r /= lamda;
        r -= ld_g(divdb + q);
        if (mode == 0) {
            out[q] = r;
            return;
        }
        const int c = (i + j + k) & 1;
        const long long pq = d.pidx(i, j, k) + (c ? d.npk() : 0);
        T ph = ld_g(phi + q);
        const bool face = i == 0 || j == 0 || k == 0 || i == d.nx - 1 || j == d.ny - 1 ||
                          k == d.nz - 1;
        if (dirichlet && face) ph = bc;
        upk[pq] = ph;
        out[pq] = mode == 2 ? r + ph * inv_dt : r;
    }
};

// ------------------------------------------------------------------- cp.async
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
// 16 bytes, or 16 zero bytes when !valid (nothing is read from gmem then)
__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ------------------------------------------------------- separable convolution
// out = sum_t w[t] x[p + t - S], symmetric taps (w[t] == w[nh-1-t]), zero outside.
template <typename T, int N>
__device__ __forceinline__ Vec<T, N> tap_sum(const Vec<T, N>* x, int stride, const T* w, int nh)
{
    const int S = nh >> 1;
    Vec<T, N> acc;
#pragma unroll
    for (int q = 0; q < N; ++q) acc.v[q] = w[S] * x[S * stride].v[q];
    for (int t = 0; t < S; ++t) {
        const Vec<T, N> a = x[t * stride];
        const Vec<T, N> b = x[(nh - 1 - t) * stride];
#pragma unroll
        for (int q = 0; q < N; ++q) acc.v[q] = fma(w[t], a.v[q] + b.v[q], acc.v[q]);
    }
    return acc;
}

// Pass along k (contiguous). Block: TK threads along k x RK rows; grid.x over rows
// (i*ny + j), grid.y over k tiles. smem: RK x (TK + 2S) vectors + taps.
template <typename T, int N, int TK, int RK, class Ld, class St>
__global__ void __launch_bounds__(TK* RK) conv_k_kernel(Ld ld, St st, Dims d, const T* __restrict__ taps,
                                                      int nh)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S = nh >> 1;
    const int W = TK + 2 * S;
    Vec<T, N>* sm = reinterpret_cast<Vec<T, N>*>(smem_raw);
    T* wsm = reinterpret_cast<T*>(sm + RK * W);
    const int tid = threadIdx.y * TK + threadIdx.x;
    for (int t = tid; t < nh; t += TK * RK) wsm[t] = taps[t];
    const long long row = (long long)blockIdx.x * RK + threadIdx.y;
    const bool live = row < (long long)d.nx * d.ny;
    const int i = live ? (int)(row / d.ny) : 0;
    const int j = live ? (int)(row % d.ny) : 0;
    const int k0 = blockIdx.y * TK;
    Vec<T, N>* srow = sm + threadIdx.y * W;
    for (int s = threadIdx.x; s < W; s += TK) {
        int kk = 0;
        srow[s] = (live && d.halo(k0 - S + s, d.nz, kk)) ? ld(i, j, kk) : vzero<T, N>();
    }
    __syncthreads();
    const int k = k0 + threadIdx.x;
    if (!live || k >= d.nz) return;
    st(i, j, k, tap_sum<T, N>(srow + threadIdx.x, 1, wsm, nh));
}

// Pass along j (AXIS 1) or i (AXIS 0). Block: TW threads along k x TY along the
// axis; tile TA outputs along the axis x TW along k. grid = (k tiles, axis tiles,
// the third coordinate). smem: (TA + 2S) x TW vectors + taps.
template <typename T, int N, int AXIS, int TW, int TY, int TA, class Ld, class St>
__global__ void __launch_bounds__(TW* TY) conv_s_kernel(Ld ld, St st, Dims d, const T* __restrict__ taps,
                                                      int nh)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S = nh >> 1;
    const int H = TA + 2 * S;
    Vec<T, N>* sm = reinterpret_cast<Vec<T, N>*>(smem_raw);
    T* wsm = reinterpret_cast<T*>(sm + H * TW);
    const int tid = threadIdx.y * TW + threadIdx.x;
    for (int t = tid; t < nh; t += TW * TY) wsm[t] = taps[t];
    const int k = blockIdx.x * TW + threadIdx.x;
    const int a0 = blockIdx.y * TA;
    const int other = blockIdx.z;
    const int len = AXIS == 0 ? d.nx : d.ny;
    const bool kin = k < d.nz;
    for (int s = threadIdx.y; s < H; s += TY) {
        int a = 0;
        Vec<T, N> v = vzero<T, N>();
        if (kin && d.halo(a0 - S + s, len, a)) v = AXIS == 0 ? ld(a, other, k) : ld(other, a, k);
        sm[s * TW + threadIdx.x] = v;
    }
    __syncthreads();
    if (!kin) return;
    for (int o = threadIdx.y; o < TA; o += TY) {
        const int a = a0 + o;
        if (a >= len) break;
        const Vec<T, N> r = tap_sum<T, N>(sm + o * TW + threadIdx.x, TW, wsm, nh);
        if (AXIS == 0) st(a, other, k, r);
        else st(other, a, k, r);
    }
}

// ---- register-window passes for a compile-time half width S (taps 2S+1) ----
// Each thread computes R consecutive outputs along the convolution axis from a
// register window of R + 2S inputs, with the taps in registers and the inputs in
// shared memory as one plane per field; this reads each staged input (R+2S)/R times
// instead of 2S+1 times.
template <typename T, int S, int R>
__device__ __forceinline__ void window_conv(const T (&x)[R + 2 * S], const T (&w)[S + 1],
                                            T (&out)[R])
{
#pragma unroll
    for (int r = 0; r < R; ++r) {
        T acc = w[S] * x[r + S];
#pragma unroll
        for (int t = 0; t < S; ++t) acc = fma(w[t], x[r + t] + x[r + 2 * S - t], acc);
        out[r] = acc;
    }
}

template <typename T, int S>
__device__ __forceinline__ void load_taps(const T* __restrict__ taps, T (&w)[S + 1])
{
#pragma unroll
    for (int t = 0; t <= S; ++t) w[t] = __ldg(taps + t);
}

// Along k (contiguous). Block TKT x RKR threads; each thread R = 4 RG consecutive k of
// one row (RG groups of 4 for the storer); tile RKR rows x R*TKT k. The halo is rounded
// up to SP = 4*ceil(S/4) so that every thread's window starts 16-byte aligned and is
// read with vector loads. Larger RG reads fewer window values per output from shared
// memory and recomputes fewer halo cells; every output is the same sum either way.
template <typename T, int N, int S, int TKT, int RKR, class Ld, class St, int RG = 1>
__device__ __forceinline__ void conv_k_win_body(const uint3 blockIdx, const dim3 gridDim, Ld ld, St st, Dims d,
                                                const T* __restrict__ taps)
{
    constexpr int R = 4 * RG;
    constexpr int TK = TKT * R;
    constexpr int SP = (S + 3) & ~3;
    constexpr int W = TK + 2 * SP;
    constexpr int XW = R + 2 * SP;  // window read by one thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);  // [N][RKR][W]
    const long long row = (long long)blockIdx.x * RKR + threadIdx.y;
    const bool live = row < (long long)d.nx * d.ny;
    const int i = live ? (int)(row / d.ny) : 0;
    const int j = live ? (int)(row % d.ny) : 0;
    const int k0 = blockIdx.y * TK;
    const int kk = k0 + threadIdx.x * R;  // this thread's first output cell (even)
    typename St::Pre pre[RG]{};
    {
        constexpr int NL = (W + TKT - 1) / TKT;
        // all reads first, then the loader's arithmetic (the Heaviside for stage 1)
        typename Ld::Raw rw[NL];
        bool ok[NL];
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.x + u * TKT;
            int k = 0;
            ok[u] = s < W && live && d.halo(k0 - SP + s, d.nz, k);
            if (ok[u]) rw[u] = ld.raw(i, j, k);
        }
        // the storer's own reads (the forcing term's fields) go out with them
#pragma unroll
        for (int g = 0; g < RG; ++g)
            if (kk + 4 * g < d.nz && live) pre[g] = st.pre(i, j, kk + 4 * g, min(4, d.nz - kk - 4 * g));
        Vec<T, N> v[NL];
#pragma unroll
        for (int u = 0; u < NL; ++u) v[u] = ok[u] ? ld.cook(rw[u]) : vzero<T, N>();
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.x + u * TKT;
            if (s < W) {
#pragma unroll
                for (int q = 0; q < N; ++q) sm[(q * RKR + threadIdx.y) * W + s] = v[u].v[q];
            }
        }
    }
    T w[S + 1];
    load_taps<T, S>(taps, w);
    __syncthreads();
    const bool act = live && kk < d.nz;
    T res[N][R];
    if (act) {
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const T* base = sm + (q * RKR + threadIdx.y) * W + threadIdx.x * R;
            T xa[XW];
            if (sizeof(T) == 4) {
#pragma unroll
                for (int t = 0; t < XW; t += 4) {
                    const float4 v4 = *reinterpret_cast<const float4*>(base + t);
                    xa[t] = v4.x; xa[t + 1] = v4.y; xa[t + 2] = v4.z; xa[t + 3] = v4.w;
                }
            } else {
#pragma unroll
                for (int t = 0; t < XW; t += 2) {
                    const double2 v2 = *reinterpret_cast<const double2*>(base + t);
                    xa[t] = v2.x; xa[t + 1] = v2.y;
                }
            }
            T x[R + 2 * S];
#pragma unroll
            for (int t = 0; t < R + 2 * S; ++t) x[t] = xa[t + SP - S];
            window_conv<T, S, R>(x, w, res[q]);
        }
    }
    if (!act) return;
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        const int kg = kk + 4 * g;
        if (kg >= d.nz) break;
        Vec<T, N> vo[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int q = 0; q < N; ++q) vo[r].v[q] = res[q][4 * g + r];
        }
        st.put4(pre[g], i, j, kg, vo, min(4, d.nz - kg));
    }
}

template <typename T, int N, int S, int TKT, int RKR, class Ld, class St, int RG = 1>
__global__ void __launch_bounds__(TKT* RKR) conv_k_win_kernel(Ld ld, St st, Dims d, const T* __restrict__ taps)
{
    conv_k_win_body<T, N, S, TKT, RKR, Ld, St, RG>(blockIdx, gridDim, ld, st, d, taps);
}

// FP32 passes of four fields convolve them in pairs (float2 in shared memory,
// __fadd2_rn / __ffma2_rn / __fmul2_rn): per component the operations of window_conv,
// so the sums are bit-identical. They run as conv_s_win_pair_kernel, held to 3 blocks
// per SM (80 registers, a few bytes spilled). Measured against the scalar form, same
// box: 4 fields 133 -> 117 us at 256^3 and 760 -> 602 us at 512x512x320; 2 fields
// 82 -> 74 and 442 -> 496 us, so the 2-field pass stays scalar.
template <typename T, int N>
constexpr bool kPairedS = sizeof(T) == 4 && N == 4;

// Along j (AXIS 1) or i (AXIS 0). Block TW x TY; each thread R consecutive outputs
// along the axis in one k column; tile TY*R along the axis x TW along k.
template <typename T, int N, int AXIS, int S, int TW, int TY, int R, class Ld, class St>
__device__ __forceinline__ void conv_s_win_body(const uint3 blockIdx, const dim3 gridDim, Ld ld, St st, Dims d, const T* __restrict__ taps)
{
    constexpr int TA = TY * R;
    constexpr int H = TA + 2 * S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sm = reinterpret_cast<T*>(smem_raw);  // [N][H][TW]
    const int k = blockIdx.x * TW + threadIdx.x;
    const int a0 = blockIdx.y * TA;
    const int other = blockIdx.z;
    const int len = AXIS == 0 ? d.nx : d.ny;
    const bool kin = k < d.nz;
    {
        constexpr int NL = (H + TY - 1) / TY;
        Vec<T, N> v[NL];
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.y + u * TY;
            int a = 0;
            v[u] = vzero<T, N>();
            if (s < H && kin && d.halo(a0 - S + s, len, a)) v[u] = AXIS == 0 ? ld(a, other, k) : ld(other, a, k);
        }
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.y + u * TY;
            if (s < H) {
                if constexpr (kPairedS<T, N>) {
                    // FP32 fields in pairs, [N/2][H][TW] of float2
#pragma unroll
                    for (int q = 0; q < N / 2; ++q)
                        reinterpret_cast<float2*>(sm)[(q * H + s) * TW + threadIdx.x] =
                            make_float2(v[u].v[2 * q], v[u].v[2 * q + 1]);
                } else {
#pragma unroll
                    for (int q = 0; q < N; ++q) sm[(q * H + s) * TW + threadIdx.x] = v[u].v[q];
                }
            }
        }
    }
    T w[S + 1];
    load_taps<T, S>(taps, w);
    __syncthreads();
    if (!kin) return;
    const int r0 = threadIdx.y * R;
    Vec<T, N> out[R];
    if constexpr (kPairedS<T, N>) {
        // window_conv of two fields at once with the paired FP32 instructions of sm_100:
        // per component the same operations, half the instructions and loads
        float2 w2[S + 1];
#pragma unroll
        for (int t = 0; t <= S; ++t) w2[t] = make_float2(w[t], w[t]);
#pragma unroll
        for (int q = 0; q < N / 2; ++q) {
            float2 x[R + 2 * S];
#pragma unroll
            for (int t = 0; t < R + 2 * S; ++t)
                x[t] = reinterpret_cast<const float2*>(sm)[(q * H + r0 + t) * TW + threadIdx.x];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 acc = __fmul2_rn(w2[S], x[r + S]);
#pragma unroll
                for (int t = 0; t < S; ++t) acc = __ffma2_rn(w2[t], __fadd2_rn(x[r + t], x[r + 2 * S - t]), acc);
                out[r].v[2 * q] = acc.x;
                out[r].v[2 * q + 1] = acc.y;
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) {
            T x[R + 2 * S];
#pragma unroll
            for (int t = 0; t < R + 2 * S; ++t) x[t] = sm[(q * H + r0 + t) * TW + threadIdx.x];
            T o[R];
            window_conv<T, S, R>(x, w, o);
#pragma unroll
            for (int r = 0; r < R; ++r) out[r].v[q] = o[r];
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int a = a0 + r0 + r;
        if (a < len) {
            if (AXIS == 0) st(a, other, k, out[r]);
            else st(other, a, k, out[r]);
        }
    }
}

template <typename T, int N, int AXIS, int S, int TW, int TY, int R, class Ld, class St>
__global__ void __launch_bounds__(TW* TY) conv_s_win_kernel(Ld ld, St st, Dims d, const T* __restrict__ taps)
{
    conv_s_win_body<T, N, AXIS, S, TW, TY, R, Ld, St>(blockIdx, gridDim, ld, st, d, taps);
}

// the paired form (kPairedS), held to 3 blocks per SM
template <typename T, int N, int AXIS, int S, int TW, int TY, int R, class Ld, class St>
__global__ void __launch_bounds__(TW* TY, 3) conv_s_win_pair_kernel(Ld ld, St st, Dims d, const T* __restrict__ taps)
{
    conv_s_win_body<T, N, AXIS, S, TW, TY, R, Ld, St>(blockIdx, gridDim, ld, st, d, taps);
}

// Fused i-axis stage with register windows (see conv_i_fit_kernel for the maths).
// First pass: RA = ceil((TA+2S)/TY) rows per thread over the four fields; second
// pass: RB = TA/TY rows per thread over the pair.
template <typename T, int S, int TW, int TY, int TA>
__device__ __forceinline__ void conv_i_fit_win_body(const uint3 blockIdx, const dim3 gridDim, const Vec<T, 4>* __restrict__ in, Vec<T, 2>* __restrict__ out, T* f1_out, T* f2_out, Dims d, const T* __restrict__ taps, T l1, T l2)
{
    constexpr int RA = (TA + 2 * S + TY - 1) / TY;
    constexpr int RB = TA / TY;
    constexpr int H2 = TY * RA;          // rows of the first pass's output (>= TA + 2S)
    constexpr int H1 = H2 + 2 * S;       // input rows
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* sin = reinterpret_cast<T*>(smem_raw);   // [4][H1][TW]
    T* smid = sin + 4 * H1 * TW;               // [2][H2][TW]
    const int k = blockIdx.x * TW + threadIdx.x;
    const int i0 = blockIdx.y * TA;
    const int j = blockIdx.z;
    const bool kin = k < d.nz;
    {
        constexpr int NL = (H1 + TY - 1) / TY;
        Vec<T, 4> v[NL];
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.y + u * TY;
            int i = 0;
            v[u] = vzero<T, 4>();
            if (s < H1 && kin && d.halo(i0 - 2 * S + s, d.nx, i)) v[u] = in[d.idx(i, j, k)];
        }
#pragma unroll
        for (int u = 0; u < NL; ++u) {
            const int s = threadIdx.y + u * TY;
            if (s < H1) {
#pragma unroll
                for (int q = 0; q < 4; ++q) sin[(q * H1 + s) * TW + threadIdx.x] = v[u].v[q];
            }
        }
    }
    T w[S + 1];
    load_taps<T, S>(taps, w);
    __syncthreads();
    {
        const int r0 = threadIdx.y * RA;
        T c[4][RA];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            T x[RA + 2 * S];
#pragma unroll
            for (int t = 0; t < RA + 2 * S; ++t) x[t] = sin[(q * H1 + r0 + t) * TW + threadIdx.x];
            window_conv<T, S, RA>(x, w, c[q]);
        }
#pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int s = r0 + r;           // first-pass row: i = i0 - S + s
            const int i = i0 - S + s;
            T pv = T(0), qv = T(0);
            // rows outside the volume are zero for the second convolution, or the
            // rows they wrap to for the periodic boundary
            const bool inside = i >= 0 && i < d.nx;
            if (kin && (inside || d.cyc)) {
                const T f1 = c[0][r] / c[1][r];
                const T f2 = c[2][r] / c[3][r];
                pv = f1 * l1 - f2 * l2;
                qv = (f1 * f1) * l1 - (f2 * f2) * l2;
                if (f1_out && inside && s >= S && s < S + TA) {
                    const long long qq = d.idx(i, j, k);
                    f1_out[qq] = f1;
                    f2_out[qq] = f2;
                }
            }
            smid[(0 * H2 + s) * TW + threadIdx.x] = pv;
            smid[(1 * H2 + s) * TW + threadIdx.x] = qv;
        }
    }
    __syncthreads();
    if (!kin) return;
    const int r0 = threadIdx.y * RB;
    T o[2][RB];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        T x[RB + 2 * S];
#pragma unroll
        for (int t = 0; t < RB + 2 * S; ++t) x[t] = smid[(q * H2 + r0 + t) * TW + threadIdx.x];
        window_conv<T, S, RB>(x, w, o[q]);
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        const int i = i0 + r0 + r;
        if (i < d.nx) {
            Vec<T, 2> v;
            v.v[0] = o[0][r];
            v.v[1] = o[1][r];
            out[d.idx(i, j, k)] = v;
        }
    }
}

template <typename T, int S, int TW, int TY, int TA>
__global__ void __launch_bounds__(TW* TY) conv_i_fit_win_kernel(const Vec<T, 4>* __restrict__ in, Vec<T, 2>* __restrict__ out, T* f1_out, T* f2_out, Dims d, const T* __restrict__ taps, T l1, T l2)
{
    conv_i_fit_win_body<T, S, TW, TY, TA>(blockIdx, gridDim, in, out, f1_out, f2_out, d, taps, l1, l2);
}

// One step of a running convolution along a march axis, on float pairs with the
// packed f32x2 pipes. acc[u] holds the partial sum of row p - S + u, where p is the
// plane being added: acc[u] <- acc[u+1] + w[u] x for u = 0 .. 2S-1 (w symmetric,
// w[u] = w[2S-u]) and acc[2S] <- w[0] x. After the step acc[0] is complete: its row
// has received w[t] x[row - S + t] for t = 0 .. 2S, in plane order. Every update
// reads a slot before the one it writes, so the window shifts with no moves and the
// 2S+1 updates of a step are independent.
template <int S>
__device__ __forceinline__ void shift_conv2(float2 (&acc)[2 * S + 1], const float2 (&w)[S + 1], float2 x)
{
#pragma unroll
    for (int u = 0; u < 2 * S; ++u) acc[u] = __ffma2_rn(w[u <= S ? u : 2 * S - u], x, acc[u + 1]);
    acc[2 * S] = __fmul2_rn(w[0], x);
}

// cp.async.wait_group with a count known only after unrolling (0 .. 15)
__device__ __forceinline__ void cp_async_wait_n(int n)
{
    switch (n) {
    case 0: cp_async_wait<0>(); break;
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    case 4: cp_async_wait<4>(); break;
    case 5: cp_async_wait<5>(); break;
    case 6: cp_async_wait<6>(); break;
    case 7: cp_async_wait<7>(); break;
    case 8: cp_async_wait<8>(); break;
    case 9: cp_async_wait<9>(); break;
    case 10: cp_async_wait<10>(); break;
    case 11: cp_async_wait<11>(); break;
    case 12: cp_async_wait<12>(); break;
    case 13: cp_async_wait<13>(); break;
    case 14: cp_async_wait<14>(); break;
    default: cp_async_wait<15>(); break;
    }
}

// taps w[0] .. w[S] of a symmetric kernel, each as a float pair (w, w), passed by value
// so that the kernel reads them from the parameter bank
template <int S>
struct TapPairs {
    float2 w[S + 1];
};

// Fused i-axis stage, marching form (FP32): the maths of conv_i_fit_kernel with no
// recomputed rows. Block: 32 threads along k x JB along j, one (j, k) column per
// thread; blockIdx.z picks a chunk of `chunk` output rows along i. A thread streams
// the input planes p = i0-2S .. i1+2S-1 of its column: each 16-byte cell goes through
// a D-plane ring in shared memory by cp.async (zero filled outside the volume,
// wrapped for the periodic boundary) and is added into the accumulators of the first
// convolution (the four fields as two f32x2 pairs). Row m = p - S of that convolution
// is then complete: (num, den, numb, denb) give f1, f2 and the pair
// (l1 f1 - l2 f2, l1 f1^2 - l2 f2^2) (zero outside the volume unless periodic), which
// is added into the accumulators of the second convolution, completing its output
// row m - S. The march takes U planes per round: one barrier per round orders the
// reads of the previous round's ring slots before they are refilled, and the U steps
// between barriers overlap one plane's division and fit with the next plane's
// accumulation. Rounding differs from the tiled kernels by summation order only: each
// row adds its 2S+1 products in plane order, where the tiled kernels add symmetric
// pairs first; f1 and f2 use the fast division (within 2 ulp).
template <int S, int JB, int D, int U, int MINB>
__device__ __forceinline__ void conv_i_fit_march_body(const uint3 blockIdx, const dim3 gridDim, const float4* __restrict__ in, float2* __restrict__ out, float* f1_out, float* f2_out, Dims d, const TapPairs<S> tp, float l1, float l2, int chunk)
{
    constexpr int L = 2 * S + 1;
    static_assert((D & (D - 1)) == 0 && D >= 2 * U && D <= 16, "ring: a power of two, >= 2U");
    __shared__ __align__(16) float4 ring[D][JB][32];
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * JB + threadIdx.y;
    const int i0 = blockIdx.z * chunk;
    const int i1 = min(i0 + chunk, d.nx);
    const bool col = k < d.nz && j < d.ny;
    const int pa = i0 - 2 * S;
    const int np = (i1 - i0) + 4 * S;
    const long long cq = (long long)j * d.nz + k;        // this column in plane 0
    const long long ps = (long long)d.ny * d.nz;         // plane stride
    float4* const mine = &ring[0][threadIdx.y][threadIdx.x];
    constexpr int SLOT = JB * 32;  // float4s between ring slots
    auto issue = [&](int n) {
        int i = 0;
        const bool ok = col && n < np && d.halo(pa + n, d.nx, i);
        const float4* src = ok ? in + (i * ps + cq) : in;
        cp_async16_zfill(mine + (n & (D - 1)) * SLOT, src, ok);
        cp_async_commit();
    };
    // planes 0 .. D-U-1 ahead of the first round
#pragma unroll
    for (int n = 0; n < D - U; ++n) issue(n);
    const float2 (&w2)[S + 1] = tp.w;
    // rows before the first one needed collect contributions and are never read
    float2 a0[L], a1[L], bq[L];
#pragma unroll
    for (int t = 0; t < L; ++t) a0[t] = a1[t] = bq[t] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int n0 = 0; n0 < np; n0 += U) {
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int n = n0 + q;
            // groups issued: planes 0 .. n0+D-U-1; plane n is complete when at most
            // D-U-1-q of them are pending
            cp_async_wait_n(D - U - 1 - q);
            if (n < np) {
                const float4 x = mine[(n & (D - 1)) * SLOT];
                shift_conv2<S>(a0, w2, make_float2(x.x, x.y));
                shift_conv2<S>(a1, w2, make_float2(x.z, x.w));
                if (n >= 2 * S) {
                    // row m = p - S of the first convolution is complete
                    const int m = pa + n - S;
                    const bool inside = m >= 0 && m < d.nx;
                    float pv = 0.f, qv = 0.f;
                    if (col && (inside || d.cyc)) {
                        // (13 taps keep the division of the kernel they used to run on)
                        const float f1 = S == 6 ? a0[0].x / a0[0].y : __fdividef(a0[0].x, a0[0].y);
                        const float f2 = S == 6 ? a1[0].x / a1[0].y : __fdividef(a1[0].x, a1[0].y);
                        pv = f1 * l1 - f2 * l2;
                        qv = (f1 * f1) * l1 - (f2 * f2) * l2;
                        if (f1_out && inside && m >= i0 && m < i1) {
                            const long long qq = m * ps + cq;
                            f1_out[qq] = f1;
                            f2_out[qq] = f2;
                        }
                    }
                    // output row m - S is complete
                    shift_conv2<S>(bq, w2, make_float2(pv, qv));
                    if (n >= 4 * S && col) out[(m - S) * ps + cq] = bq[0];
                }
            }
        }
        // every thread has read this round's slots before the next rounds refill them
        __syncthreads();
#pragma unroll
        for (int q = 0; q < U; ++q) issue(n0 + D - U + q);
    }
    cp_async_wait<0>();
}

template <int S, int JB, int D, int U, int MINB>
__global__ void __launch_bounds__(32 * JB, MINB) conv_i_fit_march_kernel(const float4* __restrict__ in, float2* __restrict__ out, float* f1_out, float* f2_out, Dims d, const TapPairs<S> tp, float l1, float l2, int chunk)
{
    conv_i_fit_march_body<S, JB, D, U, MINB>(blockIdx, gridDim, in, out, f1_out, f2_out, d, tp, l1, l2, chunk);
}

// Fused i-axis stage: K_i applied to the four stage-1 fields (H u0, H, Hb u0, Hb)
// completes num, den, numb, denb; then f1 = num/den, f2 = numb/denb, the second
// pair (l1 f1 - l2 f2, l1 f1^2 - l2 f2^2) is formed and K_i is applied to it.
// The reference's f2 = (num - k*u0)/(den - k*1) equals numb/denb by linearity of
// the convolution (k*u0 - num = k*((1-H) u0), k*1 - den = k*(1-H)).
// Tile: TA outputs along i; the first pass covers TA + 2S rows (zero outside the
// volume, which is the zero boundary of the second convolution's input).
template <typename T, int TW, int TY, int TA>
__global__ void __launch_bounds__(TW* TY) conv_i_fit_kernel(const Vec<T, 4>* __restrict__ in,
                                                          Vec<T, 2>* __restrict__ out, T* f1_out,
                                                          T* f2_out, Dims d,
                                                          const T* __restrict__ taps, int nh,
                                                          T l1, T l2)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int S = nh >> 1;
    const int H1 = TA + 4 * S;  // input rows
    const int H2 = TA + 2 * S;  // rows of the second pass's input
    Vec<T, 4>* sin = reinterpret_cast<Vec<T, 4>*>(smem_raw);
    Vec<T, 2>* smid = reinterpret_cast<Vec<T, 2>*>(sin + H1 * TW);
    T* wsm = reinterpret_cast<T*>(smid + H2 * TW);
    const int tid = threadIdx.y * TW + threadIdx.x;
    for (int t = tid; t < nh; t += TW * TY) wsm[t] = taps[t];
    const int k = blockIdx.x * TW + threadIdx.x;
    const int i0 = blockIdx.y * TA;
    const int j = blockIdx.z;
    const bool kin = k < d.nz;
    for (int s = threadIdx.y; s < H1; s += TY) {
        int i = 0;
        Vec<T, 4> v = vzero<T, 4>();
        if (kin && d.halo(i0 - 2 * S + s, d.nx, i)) v = in[d.idx(i, j, k)];
        sin[s * TW + threadIdx.x] = v;
    }
    __syncthreads();
    for (int s = threadIdx.y; s < H2; s += TY) {
        const int i = i0 - S + s;
        Vec<T, 2> m = vzero<T, 2>();
        const bool inside = i >= 0 && i < d.nx;
        if (kin && (inside || d.cyc)) {
            const Vec<T, 4> c = tap_sum<T, 4>(sin + s * TW + threadIdx.x, TW, wsm, nh);
            const T f1 = c.v[0] / c.v[1];
            const T f2 = c.v[2] / c.v[3];
            m.v[0] = f1 * l1 - f2 * l2;
            m.v[1] = (f1 * f1) * l1 - (f2 * f2) * l2;
            if (f1_out && inside && s >= S && s < S + TA) {
                const long long q = d.idx(i, j, k);
                f1_out[q] = f1;
                f2_out[q] = f2;
            }
        }
        smid[s * TW + threadIdx.x] = m;
    }
    __syncthreads();
    if (!kin) return;
    for (int o = threadIdx.y; o < TA; o += TY) {
        const int i = i0 + o;
        if (i >= d.nx) break;
        out[d.idx(i, j, k)] = tap_sum<T, 2>(smid + o * TW + threadIdx.x, TW, wsm, nh);
    }
}

// ------------------------------------------------------------------ stencils
// Spacings of the difference stencils, filled on the host (2 h and 1 / (2 h) in T: computed
// per thread in double they were most of the column kernels' instructions).
template <typename T>
struct HStep {
    T h[3], two[3], inv[3];
    int pow2;  // bit a set: 2 h of axis a is a power of two
};

// x / (2h) of the difference stencils: FP64 divides, with the reference's operations (where 2h
// is a power of two the product with its reciprocal is the same number); FP32 multiplies by
// the reciprocal, which gives the same value when 2h is a power of two (unit spacing) and is
// within 1 ulp of it otherwise, at a fraction of a division's instructions.
template <int AXIS, typename T>
__device__ __forceinline__ T over_two_h(T x, const HStep<T>& hs)
{
    if constexpr (sizeof(T) == 4) return x * hs.inv[AXIS];
    else return (hs.pow2 >> AXIS & 1) ? x * hs.inv[AXIS] : x / hs.two[AXIS];
}

// One component of image3d::grad at a point with position pos on an axis of length
// len (image3d_imp.hxx:762-838): central inside, one-sided second order on faces.
template <int AXIS, typename T>
__device__ __forceinline__ T grad_term(const T* f, long long p, long long stride, int pos, int len, const HStep<T>& hs)
{
    if (pos == 0) return over_two_h<AXIS>(T(4) * f[p + stride] - T(3) * f[p] - f[p + 2 * stride], hs);
    if (pos == len - 1) return over_two_h<AXIS>(T(3) * f[p] - T(4) * f[p - stride] + f[p - 2 * stride], hs);
    return over_two_h<AXIS>(f[p + stride] - f[p - stride], hs);
}

template <typename T>
__global__ void grad_kernel(const T* __restrict__ f, T* __restrict__ g, Dims d, HStep<T> hs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long p = d.idx(i, j, k);
    const long long n = d.n();
    g[p] = grad_term<0>(f, p, (long long)d.ny * d.nz, i, d.nx, hs);
    g[n + p] = grad_term<1>(f, p, (long long)d.nz, j, d.ny, hs);
    g[2 * n + p] = grad_term<2>(f, p, 1, k, d.nz, hs);
}

// im3d::div at one point (image3d_imp.hxx:1060-1380) with the reference's two
// stencil quirks: on the face i = X-1 (j, k inside) the x term is
// ((3f - 4f + f)/2)*hx (:1091-1099), and on the edge j = 0, k = Z-1 (i inside) the
// z term reads Z-2 twice (:1203-1213).
template <typename T>
__device__ __forceinline__ T div_point(const T* f0, const T* f1, const T* f2, const Dims& d,
                                       int i, int j, int k, HStep<T> hs)
{
    const long long p = d.idx(i, j, k);
    const long long sx = (long long)d.ny * d.nz, sy = d.nz;
    const int cx = i == 0 ? 0 : (i == d.nx - 1 ? 2 : 1);
    const int cy = j == 0 ? 0 : (j == d.ny - 1 ? 2 : 1);
    const int cz = k == 0 ? 0 : (k == d.nz - 1 ? 2 : 1);
    T tx, tz;
    if (cx == 2 && cy == 1 && cz == 1)
        tx = (T(3) * f0[p] - T(4) * f0[p - sx] + f0[p - 2 * sx]) / T(2.) * hs.h[0];
    else
        tx = grad_term<0>(f0, p, sx, i, d.nx, hs);
    const T ty = grad_term<1>(f1, p, sy, j, d.ny, hs);
    if (cx == 1 && cy == 0 && cz == 2)
        tz = (T(3) * f2[p] - T(4) * f2[p - 1] + f2[p - 1]) / hs.two[2];
    else
        tz = grad_term<2>(f2, p, 1, k, d.nz, hs);
    return tx + ty + tz;
}

// div_point for every cell, any nz: a thread owns the (j, k) column of NI planes, consecutive
// lanes consecutive k. Rows inside i and j take central x and y terms and a z term whose
// one-sided forms on the faces k = 0 and k = nz - 1 replace it by selects (the third point is
// read beside the neighbours); other rows take div_point. Every read of the NI planes comes
// before the first store. One cell per thread by div_point alone with the spacings divided per
// thread took 40 us at 171x203x117, the columns 33 us, and with HStep 31 us (FP32).
template <typename T, int NI>
__device__ __forceinline__ void div_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ v, T* __restrict__ out, Dims d, HStep<T> hs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i0 = blockIdx.z * NI;
    if (k >= d.nz || j >= d.ny) return;
    const int cnt = min(NI, d.nx - i0);
    const long long n = d.n(), plane = (long long)d.ny * d.nz, sy = d.nz;
    const T *f0 = v, *f1 = v + n, *f2 = v + 2 * n;
    const long long p0 = d.idx(i0, j, k);
    const bool jint = j >= 1 && j <= d.ny - 2;
    // the two z neighbours, or on a face the two points inward: a = k + 1 (k - 1 at the high
    // face), b = k - 1 (k + 2 at the low face, k - 2 at the high one)
    const int za = k == d.nz - 1 ? -1 : 1, zb = k == 0 ? 2 : (k == d.nz - 1 ? -2 : -1);
    T x[NI + 2], ym[NI], yp[NI], z0[NI], z1[NI], zc[NI];
#pragma unroll
    for (int t = 0; t < NI + 2; ++t) {
        const int i = i0 - 1 + t;
        x[t] = (t <= cnt + 1 && i >= 0 && i < d.nx) ? f0[p0 + (t - 1) * plane] : T(0);
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        ym[t] = yp[t] = z0[t] = z1[t] = zc[t] = T(0);
        if (t >= cnt || !jint) continue;
        const long long p = p0 + t * plane;
        ym[t] = f1[p - sy];
        yp[t] = f1[p + sy];
        zc[t] = f2[p];
        z0[t] = f2[p + za];
        z1[t] = f2[p + zb];
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        if (t >= cnt) break;
        const int i = i0 + t;
        T r;
        if (jint && i >= 1 && i <= d.nx - 2) {
            const T tx = over_two_h<0>(x[t + 2] - x[t], hs);
            const T ty = over_two_h<1>(yp[t] - ym[t], hs);
            // one division for the three forms of the z term
            const T lo = T(4) * z0[t] - T(3) * zc[t] - z1[t], hi = T(3) * zc[t] - T(4) * z0[t] + z1[t];
            r = tx + ty + over_two_h<2>(k == 0 ? lo : (k == d.nz - 1 ? hi : z0[t] - z1[t]), hs);
        } else {
            r = div_point(f0, f1, f2, d, i, j, k, hs);
        }
        out[p0 + t * plane] = r;
    }
}

template <typename T, int NI>
__global__ void __launch_bounds__(256) div_kernel(const T* __restrict__ v, T* __restrict__ out, Dims d, HStep<T> hs)
{
    div_body<T, NI>(blockIdx, gridDim, v, out, d, hs);
}

// Edge detector, GRAD branch (rsfe_splitbregman_imp.hxx:220-232, 308-313):
// g = nu / (lamda (1 + beta |grad f|^2)), evaluated in the reference's order.
template <typename T>
__global__ void edge_kernel(const T* __restrict__ f, T* __restrict__ g, Dims d, HStep<T> hs, T beta, T lamda, T nu)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long p = d.idx(i, j, k);
    const T g0 = grad_term<0>(f, p, (long long)d.ny * d.nz, i, d.nx, hs);
    const T g1 = grad_term<1>(f, p, (long long)d.nz, j, d.ny, hs);
    const T g2 = grad_term<2>(f, p, 1, k, d.nz, hs);
    T a = g0 * g0;
    a += g1 * g1;
    a += g2 * g2;
    a *= beta;
    a += T(1);
    T r = T(1);
    r /= a;
    r /= lamda;
    r *= nu;
    g[p] = r;
}

// ------------------------------------------------------------- Gauss-Seidel
template <typename T>
struct GsCoef {
    // exact reference form (double): divisions by h*h and dt
    double hx, hy, hz, dt;
    // reciprocal form (float)
    T ihx2, ihy2, ihz2, idt;
    T htilde[8];   // indexed by (cx inside) | (cy inside) << 1 | (cz inside) << 2
    // FP32: the rounding of each reciprocal, htilde_lo = 1/ht - htilde. The update
    // fma(acc, htilde, acc * htilde_lo) multiplies by 1/ht to within the final
    // rounding; acc * htilde alone would scale every update by the same relative
    // error (-2.6e-8 for 1/7), a bias of the operator that the outer iterations
    // accumulate. Unused (zero) in FP64, which keeps the reference's form.
    T htilde_lo[8];
    T bcn[4];      // bc scaled by the oblique normal for 1, 2, 3 boundary axes
    double bcnd[4];
    T bc;
    int neu;
    // FP64 forms for the residual: 1/h^2 and the diagonal 1/dt + 2/hx^2 + 2/hy^2 + 2/hz^2
    double ihx2d, ihy2d, ihz2d, diagd;
    // bit a set: h^2 of axis a (bit 3: dt) is a power of two, so that x / h^2 == x * (1 / h^2)
    // exactly
    int pow2;
    double idtd;  // 1 / dt
};

// The neighbour terms of the FP64 update divide by h^2, the own value by dt
// (poisson_imp.hxx:400). Where all of those are powers of two (P2, which the host picks by
// GsCoef::pow2) the product with the (exact) reciprocal is the same number. One form per
// kernel: with both behind a test per axis the general half-sweep of small volumes took 3.4 us
// instead of 2.9.
template <int AXIS, bool P2, typename T>
__device__ __forceinline__ double over_h2(double x, const GsCoef<T>& c)
{
    const double h = AXIS == 0 ? c.hx : AXIS == 1 ? c.hy : c.hz;
    const double r = AXIS == 0 ? c.ihx2d : AXIS == 1 ? c.ihy2d : c.ihz2d;
    return P2 ? x * r : x / (h * h);
}

template <bool P2, typename T>
__device__ __forceinline__ double over_dt(double x, const GsCoef<T>& c)
{
    return P2 ? x * c.idtd : x / c.dt;
}

// One Gauss-Seidel point value (sum of neighbour terms + b + self/dt) * htilde;
// `self_dt` is self/dt (beff mode folds u_in/dt into b and passes 0).
// r(o_i, o_j, o_k) returns the current value of a neighbour.
template <typename T, bool P2, class R>
__device__ __forceinline__ T gs_value(const GsCoef<T>& c, const Dims& d, int i, int j, int k,
                                      T b, T self, bool use_self, R r)
{
    if (!c.neu) {
        const T sx = r(1, 0, 0) + r(-1, 0, 0);
        const T sy = r(0, 1, 0) + r(0, -1, 0);
        const T sz = r(0, 0, 1) + r(0, 0, -1);
        if (std::is_same<T, double>::value) {
            double acc = over_h2<0, P2>(sx, c) + over_h2<1, P2>(sy, c) + over_h2<2, P2>(sz, c) + b;
            if (use_self) acc = acc + over_dt<P2>(self, c);
            return T(acc * (double)c.htilde[7]);
        } else {
            T acc = sx * c.ihx2 + sy * c.ihy2 + sz * c.ihz2 + b;
            if (use_self) acc += self * c.idt;
            return fma(acc, c.htilde[7], acc * c.htilde_lo[7]);
        }
    }
    const int cx = i == 0 ? 0 : (i == d.nx - 1 ? 2 : 1);
    const int cy = j == 0 ? 0 : (j == d.ny - 1 ? 2 : 1);
    const int cz = k == 0 ? 0 : (k == d.nz - 1 ? 2 : 1);
    const int nb = (cx != 1) + (cy != 1) + (cz != 1);
    const T bcn = c.bcn[nb];
    T tx, ty, tz;
    if (std::is_same<T, double>::value) {
        const double hx = c.hx, hy = c.hy, hz = c.hz;
        tx = over_h2<0, P2>(cx == 1 ? r(1, 0, 0) + r(-1, 0, 0) : (cx == 0 ? r(1, 0, 0) - bcn * hx : r(-1, 0, 0) + bcn * hx), c);
        ty = over_h2<1, P2>(cy == 1 ? r(0, 1, 0) + r(0, -1, 0) : (cy == 0 ? r(0, 1, 0) - bcn * hy : r(0, -1, 0) + bcn * hy), c);
        tz = over_h2<2, P2>(cz == 1 ? r(0, 0, 1) + r(0, 0, -1) : (cz == 0 ? r(0, 0, 1) - bcn * hz : r(0, 0, -1) + bcn * hz), c);
        double acc = (double)tx + ty + tz + b;
        if (use_self) acc = acc + over_dt<P2>(self, c);
        return T(acc * (double)c.htilde[(cx == 1) | ((cy == 1) << 1) | ((cz == 1) << 2)]);
    } else {
        const T hx = T(c.hx), hy = T(c.hy), hz = T(c.hz);
        tx = (cx == 1 ? r(1, 0, 0) + r(-1, 0, 0)
                      : (cx == 0 ? r(1, 0, 0) - bcn * hx : r(-1, 0, 0) + bcn * hx)) * c.ihx2;
        ty = (cy == 1 ? r(0, 1, 0) + r(0, -1, 0)
                      : (cy == 0 ? r(0, 1, 0) - bcn * hy : r(0, -1, 0) + bcn * hy)) * c.ihy2;
        tz = (cz == 1 ? r(0, 0, 1) + r(0, 0, -1)
                      : (cz == 0 ? r(0, 0, 1) - bcn * hz : r(0, 0, -1) + bcn * hz)) * c.ihz2;
        T acc = tx + ty + tz + b;
        if (use_self) acc += self * c.idt;
        const int m = (cx == 1) | ((cy == 1) << 1) | ((cz == 1) << 2);
        return fma(acc, c.htilde[m], acc * c.htilde_lo[m]);
    }
}

template <typename T>
__device__ __forceinline__ T gs_htilde(const GsCoef<T>& c, const Dims& d, int i, int j, int k)
{
    if (!c.neu) return c.htilde[7];
    const int ix = !(i == 0 || i == d.nx - 1), iy = !(j == 0 || j == d.ny - 1),
              iz = !(k == 0 || k == d.nz - 1);
    return c.htilde[ix | (iy << 1) | (iz << 2)];
}

// Lexicographic sweeps. Every point sees updated values at its minus neighbours and old
// ones at its plus neighbours, in the reference's i, j, k (Dir) and k, j, i (Neu) loops
// alike, so any order that keeps those dependences gives its result bit for bit.
//
// lex_tile_kernel runs all sweeps of a call in one launch, by tiles of kLexT^3 points: a
// task is one tile of one sweep. It may start when the three minus tiles have finished this
// sweep and the tile itself and the three plus tiles the previous one; done[tile] counts the
// sweeps a tile has finished. The host lists the tasks by i + j + k + 2 sweep (in tiles), a
// topological order, and the blocks take them in that order from a counter, so a task that
// a block waits for is always held by a block that runs (no co-residency is assumed). Inside
// a tile a thread owns an (i, j) column and updates k = t - i - j at step t: the tile's
// hyperplanes, one barrier each.
// What bounds it: the chain of tiles, each 3 kLexT - 2 steps of one shared-memory round trip
// and a chain of dependent additions, plus the hand-over through L2 (only the minus faces
// are read after the last wait). Measured for 5 sweeps, against one launch per hyperplane
// (bound by its launches): FP64 64^3 3804 -> 262 us, 128^3 7755 -> 411 us, 256^3 17.2 -> 1.46
// ms; FP32 64^3 3779 -> 202 us, 256^3 15.9 -> 0.86 ms.
constexpr int kLexT = 16;
constexpr int kLexH = kLexT + 2;
constexpr long long kLexWaitLimit = 1ll << 22;  // polls (under a microsecond each) before a wait gives up

// A task's tile and sweep in one word: 12 bits for i and j (up to 65535 points), 27 for k (up to
// 2^31 points), 13 for the sweep.
constexpr int kLexMaxSweeps = 1 << 13;
__host__ __device__ constexpr unsigned long long lex_task(int i, int j, int k, int sweep)
{
    return (unsigned long long)i | (unsigned long long)j << 12 | (unsigned long long)k << 24 |
           (unsigned long long)sweep << 51;
}

struct LexArgs {
    const unsigned long long* tasks;  // lex_task
    int ntasks;
    int* next;       // task counter
    int* done;       // sweeps finished per tile
    int* err;        // raised by a wait that gave up; the other blocks then stop
    int nti, ntj, ntk, lo;
};

template <typename T>
constexpr size_t lex_smem()
{
    return (size_t)(kLexH * kLexH * kLexH + kLexT * kLexT * (kLexT + 1)) * sizeof(T);
}

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int* p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits until done[w] reaches `need`; false when the limit ran out or another block failed.
__device__ __forceinline__ bool lex_wait(const LexArgs& a, int w, int need)
{
    for (long long n = 0; ld_acquire(a.done + w) < need;)
        if (++n > kLexWaitLimit || ((n & 1023) == 0 && ld_acquire(a.err) != 0)) {
            atomicExch(a.err, 1);
            return false;
        }
    return true;
}

template <typename T, bool P2>
__global__ void __launch_bounds__(kLexT* kLexT) lex_tile_kernel(T* r, const T* __restrict__ b, Dims d, GsCoef<T> c, LexArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int H = kLexH, N = kLexT;
    T* su = reinterpret_cast<T*>(smem_raw);  // [H][H][H], one halo point around the tile
    T* sb = su + H * H * H;                  // [N][N][N + 1]
    __shared__ int s_task, s_fail;
    const int tid = threadIdx.x;
    const int lj = tid % N, li = tid / N;
    const int lo = a.lo;
    const int hix = d.nx - lo, hiy = d.ny - lo, hiz = d.nz - lo;  // one past the last point updated
    for (;;) {
        if (tid == 0) {
            s_task = atomicAdd(a.next, 1);
            s_fail = 0;
        }
        __syncthreads();
        if (s_task >= a.ntasks) return;
        const unsigned long long t = a.tasks[s_task];
        const int ti = (int)(t & 0xfff), tj = (int)(t >> 12 & 0xfff), tk = (int)(t >> 24 & 0x7ffffff),
                  sw = (int)(t >> 51);
        const int i0 = lo + ti * N, j0 = lo + tj * N, k0 = lo + tk * N;
        const int tile = (ti * a.ntj + tj) * a.ntk + tk;
        const int stt[3] = {a.ntj * a.ntk, a.ntk, 1}, pos[3] = {ti, tj, tk}, len[3] = {a.nti, a.ntj, a.ntk};
        // what does not depend on this sweep's neighbours comes first: b, then (once the tile
        // and its plus tiles have finished the previous sweep) the tile and its plus faces
#pragma unroll
        for (int e = 0; e < N; ++e)
            if (i0 + e < hix && j0 + li < hiy && k0 + lj < hiz)
                sb[(e * N + li) * (N + 1) + lj] = __ldg(b + d.idx(i0 + e, j0 + li, k0 + lj));
        if (sw > 0 && tid < 4) {
            const bool has = tid == 3 || pos[tid] + 1 < len[tid];
            if (has && !lex_wait(a, tid == 3 ? tile : tile + stt[tid], sw)) s_fail = 1;
        }
        __syncthreads();
        if (s_fail) return;
        // (values of other blocks are read through L2)
        {
            T v[N + 3];
#pragma unroll
            for (int e = 0; e < N; ++e) {
                v[e] = T(0);
                if (i0 + e < d.nx && j0 + li < d.ny && k0 + lj < d.nz) v[e] = __ldcg(r + d.idx(i0 + e, j0 + li, k0 + lj));
            }
            v[N] = v[N + 1] = v[N + 2] = T(0);
            if (i0 + N < d.nx && j0 + li < d.ny && k0 + lj < d.nz) v[N] = __ldcg(r + d.idx(i0 + N, j0 + li, k0 + lj));
            if (i0 + li < d.nx && j0 + N < d.ny && k0 + lj < d.nz) v[N + 1] = __ldcg(r + d.idx(i0 + li, j0 + N, k0 + lj));
            if (i0 + li < d.nx && j0 + lj < d.ny && k0 + N < d.nz) v[N + 2] = __ldcg(r + d.idx(i0 + li, j0 + lj, k0 + N));
#pragma unroll
            for (int e = 0; e <= N; ++e) su[((e + 1) * H + li + 1) * H + lj + 1] = v[e];
            su[((li + 1) * H + N + 1) * H + lj + 1] = v[N + 1];
            su[((li + 1) * H + lj + 1) * H + N + 1] = v[N + 2];
        }
        // the minus faces: this sweep's values
        if (tid < 3 && pos[tid] > 0 && !lex_wait(a, tile - stt[tid], sw + 1)) s_fail = 1;
        __syncthreads();
        if (s_fail) return;
        {
            T v0 = T(0), v1 = T(0), v2 = T(0);
            if (i0 > 0 && j0 + li < d.ny && k0 + lj < d.nz) v0 = __ldcg(r + d.idx(i0 - 1, j0 + li, k0 + lj));
            if (j0 > 0 && i0 + li < d.nx && k0 + lj < d.nz) v1 = __ldcg(r + d.idx(i0 + li, j0 - 1, k0 + lj));
            if (k0 > 0 && i0 + li < d.nx && j0 + lj < d.ny) v2 = __ldcg(r + d.idx(i0 + li, j0 + lj, k0 - 1));
            su[(li + 1) * H + lj + 1] = v0;
            su[(li + 1) * H * H + lj + 1] = v1;
            su[((li + 1) * H + lj + 1) * H] = v2;
        }
        __syncthreads();
        const int i = i0 + li, j = j0 + lj;
        const bool col = i < hix && j < hiy;
        T* p = su + ((li + 1) * H + lj + 1) * H + 1;  // this column, at the k of the next update
        const T* pb = sb + (li * N + lj) * (N + 1);
        // old values of the next update, read a step ahead of it (the plus neighbours change
        // one step after it at the earliest)
        T zm = p[-1], self = p[0], zp = p[1], xp = p[H * H], yp = p[H], bv = pb[0];
        const int kn = min(N, hiz - k0);
        const int s0 = li + lj;
        for (int step = 0; step < 3 * N - 2; ++step) {
            const int lk = step - s0;
            if (col && lk >= 0 && lk < kn) {
                const T xm = p[-H * H], ym = p[-H];
                auto rd = [&](int oi, int oj, int ok) {
                    return oi > 0 ? xp : oi < 0 ? xm : oj > 0 ? yp : oj < 0 ? ym : ok > 0 ? zp : zm;
                };
                const T v = gs_value<T, P2>(c, d, i, j, k0 + lk, bv, self, true, rd);
                *p = v;
                ++p;
                ++pb;
                zm = v;
                self = zp;
                if (lk + 1 < N) {
                    zp = p[1];
                    xp = p[H * H];
                    yp = p[H];
                    bv = *pb;
                }
            }
            __syncthreads();
        }
        // back to global memory, rows of k
#pragma unroll
        for (int e = 0; e < N; ++e)
            if (i0 + e < hix && j0 + li < hiy && k0 + lj < hiz)
                r[d.idx(i0 + e, j0 + li, k0 + lj)] = su[((e + 1) * H + li + 1) * H + lj + 1];
        __threadfence();
        __syncthreads();
        if (tid == 0) st_release(a.done + tile, sw + 1);
    }
}

// One hyperplane i + j + k = s of a lexicographic sweep: its unknowns are independent of each
// other given the planes s - 1 (already updated) and s + 1 (not yet). Threads cover (i, j). For
// calls that have no memory for lex_tile_kernel's list; bound by its launches, one per
// hyperplane.
template <typename T>
__global__ void lex_plane_kernel(T* r, const T* __restrict__ b, Dims d, GsCoef<T> c, int s, int lo, int i_begin, int j_begin)
{
    const int j = j_begin + blockIdx.x * blockDim.x + threadIdx.x;
    const int i = i_begin + blockIdx.y * blockDim.y + threadIdx.y;
    const int hix = d.nx - lo, hiy = d.ny - lo, hiz = d.nz - lo;
    if (i >= hix || j >= hiy) return;
    const int k = s - i - j;
    if (k < lo || k >= hiz) return;
    const long long p = d.idx(i, j, k);
    auto rd = [&](int oi, int oj, int ok) { return r[d.idx(i + oi, j + oj, k + ok)]; };
    r[p] = gs_value<T, false>(c, d, i, j, k, b[p], r[p], true, rd);
}

// Dirichlet boundary assignment of DirGaussSeidel (poisson_imp.hxx:366-391).
template <typename T>
__global__ void dir_faces_kernel(T* r, Dims d, T bc)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    if (i == 0 || j == 0 || k == 0 || i == d.nx - 1 || j == d.ny - 1 || k == d.nz - 1)
        r[d.idx(i, j, k)] = bc;
}

// The (vector group g, row j) pairs of a block of planes, flattened over the grid's x
// blocks, so that no lane idles when a row's `groups` are not a multiple of blockDim.x
// (40 groups at nz = 320 left 24 of every 64 lanes idle). A power-of-two number of
// groups (nz = 256) takes shifts instead of the division.
__device__ __forceinline__ void flat_pair(const uint3 blockIdx, unsigned groups, int& g, int& j)
{
    const unsigned lin = (blockIdx.x * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
    if ((groups & (groups - 1)) == 0) {
        g = (int)(lin & (groups - 1));
        j = (int)(lin >> (__ffs((int)groups) - 1));
    } else {
        g = (int)(lin % groups);
        j = (int)(lin / groups);
    }
}

// Vectorised red-black half sweep: one thread per group of W = 16/sizeof(T)
// consecutive packed points (m0 .. m0+W-1) of row j, marching over NI planes of i.
// All points of a packed row share the parity of k, so their k neighbours are the
// other colour at (m-1, m) (k even) or (m, m+1) (k odd): one 16-byte vector plus one
// scalar. The i neighbours come from a register window of vectors along i.
// General form: the point's own old value (use_self or omega != 1) and both boundary
// rules; the residual solve with omega 1 runs rb_march_kernel instead.
// reverse: the blocks take the planes of i from the last to the first, so that a
// half-sweep following one in the other direction starts on the planes that are still
// in L2. (Without the lower bound of one block per SM the compiler keeps to fewer registers:
// 200^3 FP64 36.0 -> 36.5 us, Neumann 60.9 -> 62.2.)
template <typename T, int NI, bool P2>
__global__ void __launch_bounds__(128, 1) rb_half_vec_kernel(T* __restrict__ U, const T* B, Dims d, GsCoef<T> c, int color, int use_self, T omega, int reverse)
{
    typedef long long IX;
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    // Launched as a programmatic dependent of the previous half-sweep: wait until its
    // writes are visible, then let the next half-sweep's blocks be scheduled while this
    // one drains (both are no-ops in an ordinary launch).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    int g, j;
    flat_pair(blockIdx, (unsigned)(d.hz() / W), g, j);
    const int i0 = (reverse ? gridDim.z - 1 - blockIdx.z : blockIdx.z) * NI;
    const int hz = d.hz();
    const int m0 = g * W;
    if (m0 >= hz || j >= d.ny) return;
    const IX plane = (IX)d.ny * hz;
    const IX npk = plane * d.nx;
    T* own = U + (color ? npk : 0);
    const T* oth = U + (color ? 0 : npk);
    const T* bb = B + (color ? npk : 0);
    const bool jint = j >= 1 && j <= d.ny - 2;
    const IX q0 = ((IX)i0 * d.ny + j) * hz + m0;
    const bool relax = omega != T(1);
    // Every load of the NI planes is issued before the first store: the stores go to
    // the same array, so loads placed after one could not be moved ahead of it and each
    // thread would pay one memory round trip per plane.
    VV o[NI + 2], ymv[NI], ypv[NI], bvv[NI], sfv[NI];
    T exv[NI];
#pragma unroll
    for (int t = 0; t < NI + 2; ++t) {
        const int i = i0 - 1 + t;
        if (i >= 0 && i < d.nx) o[t] = *reinterpret_cast<const VV*>(oth + q0 + (IX)(t - 1) * plane);
        else o[t] = VV{};
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        const IX q = q0 + (IX)t * plane;
        const int par = (i + j + color) & 1;
        ymv[t] = ypv[t] = bvv[t] = sfv[t] = VV{};
        exv[t] = T(0);
        if (jint && i >= 1 && i <= d.nx - 2) {
            ymv[t] = *reinterpret_cast<const VV*>(oth + q - hz);
            ypv[t] = *reinterpret_cast<const VV*>(oth + q + hz);
            bvv[t] = *reinterpret_cast<const VV*>(bb + q);
            // the k neighbour not in the centre vector: m0-1 (k even) or m0+W (k odd)
            const bool e_ok = par ? (m0 + W < hz) : (m0 >= 1);
            if (e_ok) exv[t] = oth[par ? q + W : q - 1];
            if (use_self || relax) sfv[t] = *reinterpret_cast<const VV*>(own + q);
        }
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        if (i >= d.nx) break;
        const IX q = q0 + (IX)t * plane;
        const int par = (i + j + color) & 1;
        const bool rowint = jint && i >= 1 && i <= d.nx - 2;
        if (rowint) {
            const VV ym = ymv[t];
            const VV yp = ypv[t];
            const VV bv = bvv[t];
            const T extra = exv[t];
            const VV self = sfv[t];
            VV outv = self;
            bool all = true;
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                const int k = 2 * (m0 + cc) + par;
                const bool in = k >= 1 && k <= d.nz - 2;
                if (!in) {
                    all = false;
                    continue;
                }
                const T ctr = VT::get(o[t + 1], cc);
                const T kn = par ? (cc + 1 < W ? VT::get(o[t + 1], cc + 1) : extra)
                                 : (cc >= 1 ? VT::get(o[t + 1], cc - 1) : extra);
                const T sz = ctr + kn;
                const T sy = VT::get(ym, cc) + VT::get(yp, cc);
                const T sx = VT::get(o[t], cc) + VT::get(o[t + 2], cc);
                const T b = VT::get(bv, cc);
                const T sf = VT::get(self, cc);
                T v;
                if (std::is_same<T, double>::value) {
                    double acc = over_h2<0, P2>(sx, c) + over_h2<1, P2>(sy, c) + over_h2<2, P2>(sz, c) + b;
                    if (use_self) acc = acc + over_dt<P2>(sf, c);
                    v = T(acc * (double)c.htilde[7]);
                } else {
                    T acc = fma(sx, c.ihx2, fma(sy, c.ihy2, fma(sz, c.ihz2, b)));
                    if (use_self) acc = fma(sf, c.idt, acc);
                    v = fma(acc, c.htilde[7], acc * c.htilde_lo[7]);
                }
                if (relax) v = sf + omega * (v - sf);
                VT::set(outv, cc, v);
            }
            if (all) {
                *reinterpret_cast<VV*>(own + q) = outv;
            } else {
#pragma unroll
                for (int cc = 0; cc < W; ++cc) {
                    const int k = 2 * (m0 + cc) + par;
                    if (k >= 1 && k <= d.nz - 2) own[q + cc] = VT::get(outv, cc);
                }
            }
        }
        if (c.neu) {
            // Neumann: boundary points (faces of i, j or k) through the generic rule
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                const int k = 2 * (m0 + cc) + par;
                if (k >= d.nz) continue;
                if (rowint && k >= 1 && k <= d.nz - 2) continue;
                auto rd = [&](int oi, int oj, int ok) { return oth[d.pidx(i + oi, j + oj, k + ok)]; };
                const T sf = own[q + cc];
                T v = gs_value<T, P2>(c, d, i, j, k, bb[q + cc], sf, use_self != 0, rd);
                if (relax) v = sf + omega * (v - sf);
                own[q + cc] = v;
            }
        }
    }
}

// The W cells of one packed row group: neighbour sums in, updated values out. FP32 runs
// on the paired FP32 instructions (per component the scalar operations).
template <typename T>
struct RbRow;
template <>
struct RbRow<float> {
    template <bool>
    static __device__ __forceinline__ float4 update(const GsCoef<float>& c, const float4& xm, const float4& xp,
                                                    const float4& ym, const float4& yp, const float4& zc,
                                                    const float4& zn, const float4& b, const float (&ht)[4],
                                                    const float (&hl)[4], const bool (&)[4])
    {
        auto pair = [&](float2 a0, float2 a1, float2 b0, float2 b1, float2 c0, float2 c1, float2 bv, float2 h,
                        float2 l) {
            const float2 sx = __fadd2_rn(a0, a1), sy = __fadd2_rn(b0, b1), sz = __fadd2_rn(c0, c1);
            const float2 acc = __ffma2_rn(sx, make_float2(c.ihx2, c.ihx2),
                                          __ffma2_rn(sy, make_float2(c.ihy2, c.ihy2),
                                                     __ffma2_rn(sz, make_float2(c.ihz2, c.ihz2), bv)));
            return __ffma2_rn(acc, h, __fmul2_rn(acc, l));
        };
        const float2 lo = pair(make_float2(xm.x, xm.y), make_float2(xp.x, xp.y), make_float2(ym.x, ym.y),
                               make_float2(yp.x, yp.y), make_float2(zc.x, zc.y), make_float2(zn.x, zn.y),
                               make_float2(b.x, b.y), make_float2(ht[0], ht[1]), make_float2(hl[0], hl[1]));
        const float2 hi = pair(make_float2(xm.z, xm.w), make_float2(xp.z, xp.w), make_float2(ym.z, ym.w),
                               make_float2(yp.z, yp.w), make_float2(zc.z, zc.w), make_float2(zn.z, zn.w),
                               make_float2(b.z, b.w), make_float2(ht[2], ht[3]), make_float2(hl[2], hl[3]));
        return make_float4(lo.x, lo.y, hi.x, hi.y);
    }
};
template <>
struct RbRow<double> {
    template <bool P2>
    static __device__ __forceinline__ double2 update(const GsCoef<double>& c, const double2& xm, const double2& xp,
                                                     const double2& ym, const double2& yp, const double2& zc,
                                                     const double2& zn, const double2& b, const double (&ht)[2],
                                                     const double (&)[2], const bool (&live)[2])
    {
        auto one = [&](double sx, double sy, double sz, double bv, double h, bool lv) {
            // (the neighbours of a cell on a face or past the row are often 0, which the division
            // takes a slow path for)
            if constexpr (!P2) {
                sx = lv ? sx : 1.;
                sy = lv ? sy : 1.;
                sz = lv ? sz : 1.;
            }
            return (over_h2<0, P2>(sx, c) + over_h2<1, P2>(sy, c) + over_h2<2, P2>(sz, c) + bv) * h;
        };
        return make_double2(one(xm.x + xp.x, ym.x + yp.x, zc.x + zn.x, b.x, ht[0], live[0]),
                            one(xm.y + xp.y, ym.y + yp.y, zc.y + zn.y, b.y, ht[1], live[1]));
    }
};

// 16-byte accesses with an L2 eviction policy (createpolicy).
__device__ __forceinline__ uint64_t l2_evict_first()
{
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_last()
{
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float4 ld16_hint(const float4* a, uint64_t policy)
{
    float4 v;
    asm volatile("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(a), "l"(policy));
    return v;
}
__device__ __forceinline__ void st16_hint(float4* a, const float4& v, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;"
                 ::"l"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(policy)
                 : "memory");
}

// Boundary rules of the residual solve's half-sweep: Dirichlet; Neumann with value 0 (the
// segmentation loop's); Neumann with any value.
enum { RB_DIR = 0, RB_NEU0 = 1, RB_NEU = 2 };

// The update of the group of cells m0 .. m0+W-1 of row (i, j): xm, xp, ym, yp the groups of the
// other colour around it (0 where there is none), xc the one at its place, extra the cell
// beside it that is the missing k neighbour (par = parity of the row's cells), bv b_eff.
template <typename T, int BC, bool P2>
__device__ __forceinline__ typename V16<T>::type rb_group(const GsCoef<T>& c, const Dims& d, int i, int j, int m0, int par,
                                                          typename V16<T>::type xm, const typename V16<T>::type& xc,
                                                          typename V16<T>::type xp, typename V16<T>::type ym,
                                                          typename V16<T>::type yp, T extra,
                                                          const typename V16<T>::type& bv)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    constexpr bool NEU = BC != RB_DIR;
    VV zc = xc, zn;
#pragma unroll
    for (int cc = 0; cc < W; ++cc)
        VT::set(zn, cc, par ? (cc + 1 < W ? VT::get(xc, cc + 1) : extra) : (cc >= 1 ? VT::get(xc, cc - 1) : extra));
    // cells of the group on the faces k = 0 and k = nz - 1, and past the row
    const bool first_k = par == 0 && m0 == 0;         // cell 0 has k = 0
    const int last = ((d.nz - 1 - par) >> 1) - m0;    // the last cell with k < nz
    const bool last_k = ((d.nz - 1 - par) & 1) == 0;  // ... and whether its k is nz - 1
    T ht[W], hl[W];
    if constexpr (!NEU) {
#pragma unroll
        for (int cc = 0; cc < W; ++cc) {
            ht[cc] = c.htilde[7];
            hl[cc] = c.htilde_lo[7];
        }
    } else {
        const int cx = i == 0 ? 0 : (i == d.nx - 1 ? 2 : 1), cy = j == 0 ? 0 : (j == d.ny - 1 ? 2 : 1);
        const int nb = (cx != 1) + (cy != 1), m = (cx == 1) | ((cy == 1) << 1);
        const T hin = c.htilde[m | 4], hon = c.htilde[m], lin = c.htilde_lo[m | 4], lon = c.htilde_lo[m];
#pragma unroll
        for (int cc = 0; cc < W; ++cc) {
            const bool at0 = cc == 0 && first_k, at1 = last_k && cc == last;
            ht[cc] = at0 || at1 ? hon : hin;
            hl[cc] = at0 || at1 ? lon : lin;
            if constexpr (BC == RB_NEU) {
                const T bcn = c.bcn[at0 || at1 ? nb + 1 : nb];
                if (cx == 0) VT::set(xm, cc, -(bcn * T(c.hx)));
                if (cx == 2) VT::set(xp, cc, bcn * T(c.hx));
                if (cy == 0) VT::set(ym, cc, -(bcn * T(c.hy)));
                if (cy == 2) VT::set(yp, cc, bcn * T(c.hy));
                if (at0) VT::set(zn, cc, -(bcn * T(c.hz)));
                if (at1) {
                    if (par) VT::set(zn, cc, bcn * T(c.hz));
                    else VT::set(zc, cc, bcn * T(c.hz));
                }
            } else if (at1) {
                if (par) VT::set(zn, cc, T(0));
                else VT::set(zc, cc, T(0));
            }
        }
    }
    bool live[W];  // cells that keep the formula's value (read by the form with divisions only)
#pragma unroll
    for (int cc = 0; cc < W; ++cc)
        live[cc] = cc <= last && (NEU || !((cc == 0 && first_k) || (last_k && cc == last)));
    VV v = RbRow<T>::template update<P2>(c, xm, xp, ym, yp, zc, zn, bv, ht, hl, live);
#pragma unroll
    for (int cc = 0; cc < W; ++cc) {
        if (!NEU && ((cc == 0 && first_k) || (last_k && cc == last))) VT::set(v, cc, c.bc);
        if (cc > last) VT::set(v, cc, T(0));
    }
    return v;
}

// Half-sweep of the residual solve: own value and relaxation out of the way, the updated
// colour `own` and the other colour `oth` as separate pointers, so that no store holds a
// load back. Only `own` is __restrict__: the previous launch may still be writing `oth` (and the
// first one's, b_eff) while this one's blocks are resident, so their loads must stay ordinary
// ones that the wait below orders. One thread per group of W = 16/sizeof(T) packed cells of row j, marching over
// NI planes of i with the next plane's reads in flight. Every cell of a group is computed
// by the interior formula, without a test per cell:
//  * the k neighbours are the group itself and the group shifted by one cell (the parity of
//    the row picks the direction);
//  * Dirichlet: the cells on the k faces, which the interior formula does not apply to,
//    are written with their value again (bc; the padding after the row stays 0), and rows
//    on the other faces have no work;
//  * Neumann: a missing neighbour is replaced before the sum by the ghost value -bcn h (low
//    face) or +bcn h (high face) of NeuGaussSeidel (poisson_imp.hxx:23-336), which is 0 for
//    RB_NEU0, and the diagonal is the face's.
// first: the launch follows the kernel that wrote b_eff, so b_eff is read only after the
// wait; later half-sweeps read it before (it was complete when the launch they depend on
// passed its own wait), which overlaps the previous half-sweep's tail.
// FP32: b_eff is read with evict_first and u written with evict_last, so that u (67 MB at
// 256^3, which with b_eff's 67 MB exceeds the 126 MB L2) stays in L2 between half-sweeps:
// 17.3 -> 14.6 us at 256^3. FP64 measured slower with the policies (4.9 -> 5.5 us at 128^3).
// What bounds it: L2 bandwidth (about 15 B per cell from NI + 2 planes per NI and the rows
// around a block), DRAM for b_eff. Measured us per half-sweep in sequence, against the
// general kernel's form of it (54 instructions per cell): 256^3 FP32 17.0 -> 14.0,
// 512x512x320 88.6 -> 83.4, 160^3 5.2 -> 4.0, 171x203x117 FP32 Neumann 14.0 -> 5.7,
// 128^3 FP64 7.5 -> 4.7 and 200^3 FP64 28.4 -> 17.3 (no division per cell, over_h2), with
// spacings that need the divisions 7.6 -> 7.2 and 28.4 -> 27.8.
template <typename T, int NI, int BC, typename IX, bool P2 = false>
__device__ __forceinline__ void rb_march_body(const uint3 blockIdx, const dim3 gridDim, T* __restrict__ own,
                                              const T* oth, const T* bb, const Dims& d,
                                              const GsCoef<T>& c, int color, int reverse, int first)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    constexpr bool NEU = BC != RB_DIR;
    int g, j;
    const int hz = d.hz();
    flat_pair(blockIdx, (unsigned)(hz / W), g, j);
    const int lo = NEU ? 0 : 1;
    const int ib = (int)(reverse ? gridDim.z - 1 - blockIdx.z : blockIdx.z) * NI;
    const int i0 = ib < lo ? lo : ib, i1 = min(ib + NI, d.nx - lo);
    const int m0 = g * W;
    const bool live = j >= lo && j < d.ny - lo && i0 < i1;
    const IX plane = (IX)d.ny * hz;
    const IX q0 = ((IX)i0 * d.ny + j) * hz + m0;
    const T* pb = bb + q0;
    auto ld_b = [](const T* p) {
        if constexpr (sizeof(T) == 4) return ld16_hint(reinterpret_cast<const VV*>(p), l2_evict_first());
        else return *reinterpret_cast<const VV*>(p);
    };
    VV bn = VV{};
    if (!first && live) bn = ld_b(pb);
    // Launched as a programmatic dependent of the previous half-sweep: wait until its
    // writes are visible, then let the next half-sweep's blocks be scheduled while this
    // one drains (both are no-ops in an ordinary launch).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!live) return;
    if (first) bn = ld_b(pb);
    const T* po = oth + q0;
    T* pw = own + q0;
    const int cy = j == 0 ? 0 : (j == d.ny - 1 ? 2 : 1);
    const bool has_ym = !NEU || cy != 0, has_yp = !NEU || cy != 2;
    int par = (i0 + j + color) & 1;
    // the reads of one plane: the group's y neighbours and the k neighbour outside the group
    VV xm = VV{}, xc, ymn = VV{}, ypn = VV{};
    T en = T(0);
    auto side = [&](const T* p, int pr) {
        if (has_ym) ymn = *reinterpret_cast<const VV*>(p - hz);
        if (has_yp) ypn = *reinterpret_cast<const VV*>(p + hz);
        const bool e_ok = pr ? m0 + W < hz : m0 >= 1;
        en = e_ok ? p[pr ? W : -1] : T(0);
    };
    if (!NEU || i0 >= 1) xm = *reinterpret_cast<const VV*>(po - plane);
    xc = *reinterpret_cast<const VV*>(po);
    side(po, par);
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        if (i >= i1) break;
        const VV ym = ymn, yp = ypn, bv = bn;
        VV xp = VV{};
        const T extra = en;
        if (!NEU || i + 1 < d.nx) xp = *reinterpret_cast<const VV*>(po + plane);
        if (t + 1 < NI && i + 1 < i1) {
            side(po + plane, par ^ 1);
            pb += plane;
            bn = ld_b(pb);
        }
        const VV v = rb_group<T, BC, P2>(c, d, i, j, m0, par, xm, xc, xp, ym, yp, extra, bv);
        if constexpr (sizeof(T) == 4) st16_hint(reinterpret_cast<VV*>(pw), v, l2_evict_last());
        else *reinterpret_cast<VV*>(pw) = v;
        pw += plane;
        po += plane;
        xm = xc;
        xc = xp;
        par ^= 1;
    }
}

template <typename T, int NI, int BC, int MINB, typename IX, bool P2>
__global__ void __launch_bounds__(128, MINB) rb_march_kernel(T* __restrict__ own, const T* oth, const T* bb, Dims d, GsCoef<T> c, int color, int reverse, int first)
{
    rb_march_body<T, NI, BC, IX, P2>(blockIdx, gridDim, own, oth, bb, d, c, color, reverse, first);
}

// ---- all sweeps between two residual checks of a small volume in one launch ----
// One cluster of kRbCluster blocks holds the whole solve state in shared memory: block r the
// planes r P .. of both colours of u, one halo plane on either side, and b_eff. A half-sweep
// updates a block's own planes (rb_group: the numbers of rb_march_kernel) and writes the first
// and last of them into the neighbours' halos as well (distributed shared memory); a cluster
// barrier ends it. What bounds it: the barrier and the chain of a thread's planes; a launch per
// half-sweep cannot come below 2.4 us. us per half-sweep: 48x44x40 FP32 2.42 -> 0.90, Neumann
// 6.2 -> 0.92, 64^3 2.44 -> 1.64, 48x44x40 FP64 2.68 -> 1.41 (256, 384, 768 and 1024 threads
// measured slower).
constexpr int kRbCluster = 16, kRbClThreads = 512;

template <typename T>
__host__ __device__ inline size_t rb_cluster_smem(const Dims& d)
{
    const int P = (d.nx + kRbCluster - 1) / kRbCluster;
    return (size_t)d.ny * d.hz() * (2 * (P + 2) + 2 * P) * sizeof(T);
}

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// the 16 bytes v to the place of `p` (this block's shared memory) in block `rank` of the cluster
template <typename VV>
__device__ __forceinline__ void st16_cluster(const void* p, unsigned rank, const VV& v)
{
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    const float4 f = *reinterpret_cast<const float4*>(&v);
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(r), "f"(f.x), "f"(f.y), "f"(f.z), "f"(f.w)
                 : "memory");
}

template <typename T, int BC, bool P2>
__global__ void __launch_bounds__(kRbClThreads, 1) rb_cluster_kernel(T* __restrict__ U, const T* __restrict__ B, Dims d,
                                                                     GsCoef<T> c, int sweeps)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    constexpr bool NEU = BC != RB_DIR;
    constexpr int lo = NEU ? 0 : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    const unsigned rank = cluster_rank();
    const int hz = d.hz(), groups = hz / W;
    const int P = (d.nx + kRbCluster - 1) / kRbCluster;
    const int i0 = (int)rank * P, np = max(0, min(P, d.nx - i0));  // own planes i0 .. i0+np-1
    const int cells = d.ny * hz;                                  // of a plane and colour
    const long long npk = d.npk();
    T* su[2] = {reinterpret_cast<T*>(smem_raw), reinterpret_cast<T*>(smem_raw) + (size_t)(P + 2) * cells};
    T* sb[2] = {su[1] + (size_t)(P + 2) * cells, su[1] + (size_t)(P + 2) * cells + (size_t)P * cells};
    // plane p of su is i0 - 1 + p; planes outside the volume are 0
    const int vecs = cells / W;
    for (int col = 0; col < 2; ++col) {
        for (int q = tid; q < (np + 2) * vecs; q += kRbClThreads) {
            const int p = q / vecs, i = i0 - 1 + p;
            VV v = VV{};
            if (i >= 0 && i < d.nx) v = reinterpret_cast<const VV*>(U + col * npk + (long long)i * cells)[q - p * vecs];
            reinterpret_cast<VV*>(su[col])[q] = v;
        }
        for (int q = tid; q < np * vecs; q += kRbClThreads)
            reinterpret_cast<VV*>(sb[col])[q] = reinterpret_cast<const VV*>(B + col * npk + (long long)i0 * cells)[q];
    }
    // columns (row j, group g) times segments of the planes, so that most threads have work
    const int rows = d.ny - 2 * lo, cols = rows * groups;
    const int segs = max(1, min(np, kRbClThreads / max(cols, 1))), len = (np + segs - 1) / segs;
    // planes of this block's neighbours below and above (their halos receive the edges)
    const bool below = rank > 0 && np > 0, above = (int)rank + 1 < kRbCluster && i0 + np < d.nx;
    // a thread's items tid, tid + threads, ...; the first one's place is worked out once
    auto place = [&](int q, int& j, int& m0, int& pa, int& pb) {
        const int sg = q / cols, r = q - sg * cols, jr = r / groups;
        j = lo + jr;
        m0 = (r - jr * groups) * W;
        pa = max(sg * len, lo - i0);
        pb = min(min((sg + 1) * len, np), d.nx - lo - i0);
    };
    int j0 = 0, mm0 = 0, pa0 = 0, pb0 = 0;
    if (tid < cols * segs) place(tid, j0, mm0, pa0, pb0);
    cluster_barrier();  // every block has read U and runs
    for (int h = 0; h < 2 * sweeps; ++h) {
        const int color = h & 1;
        T* own = color ? su[1] : su[0];
        const T* oth = color ? su[0] : su[1];
        const T* bb = color ? sb[1] : sb[0];
        for (int q = tid; q < cols * segs; q += kRbClThreads) {
            int j = j0, m0 = mm0, pa = pa0, pb = pb0;
            if (q != tid) place(q, j, m0, pa, pb);
            if (pa >= pb) continue;
            const int at = j * hz + m0;
            VV xm = *reinterpret_cast<const VV*>(oth + pa * cells + at);
            VV xc = *reinterpret_cast<const VV*>(oth + (pa + 1) * cells + at);
            int par = (i0 + pa + j + color) & 1;
            for (int p = pa; p < pb; ++p) {
                const T* po = oth + (p + 1) * cells + at;
                const VV xp = *reinterpret_cast<const VV*>(po + cells);
                VV ym = VV{}, yp = VV{};
                if (!NEU || j > 0) ym = *reinterpret_cast<const VV*>(po - hz);
                if (!NEU || j < d.ny - 1) yp = *reinterpret_cast<const VV*>(po + hz);
                const bool e_ok = par ? m0 + W < hz : m0 >= 1;
                const T extra = e_ok ? po[par ? W : -1] : T(0);
                const VV bv = *reinterpret_cast<const VV*>(bb + p * cells + at);
                const VV v = rb_group<T, BC, P2>(c, d, i0 + p, j, m0, par, xm, xc, xp, ym, yp, extra, bv);
                T* pw = own + (p + 1) * cells + at;
                *reinterpret_cast<VV*>(pw) = v;
                // plane 0 is the neighbour below's halo P + 1 (it holds P planes), plane np - 1
                // the neighbour above's halo 0
                if (p == 0 && below) st16_cluster(own + (size_t)(P + 1) * cells + at, rank - 1, v);
                if (p == np - 1 && above) st16_cluster(own + at, rank + 1, v);
                xm = xc;
                xc = xp;
                par ^= 1;
            }
        }
        cluster_barrier();
    }
    for (int col = 0; col < 2; ++col)
        for (int q = tid; q < np * vecs; q += kRbClThreads)
            reinterpret_cast<VV*>(U + col * npk + (long long)i0 * cells)[q] = reinterpret_cast<const VV*>(su[col])[q + vecs];
}

// FP64 residual of (1/dt - Lap) u = b_eff over the unknowns, and sum b_eff^2 when want_beff;
// blockIdx.z covers (plane block, colour). The walk of rb_march_kernel: a thread takes a group
// of W packed cells over ni <= NI planes of i, every cell by the interior formula
//   r = sum of neighbour terms + b_eff - diag * u,  diag = 1/dt + sum_a c_a / h_a^2,
// with c_a = 2 inside; on a Neumann face the missing neighbour is the ghost value of
// rb_group and c_a = 1, and cells that are no unknowns (Dirichlet faces, padding) count 0.
// What bounds it: conversions to FP64 (about 5 per cell; a value is converted once and kept
// for the planes that read it) and the reads. us against per-cell face tests with a generic
// boundary path (88 instructions per cell): 256^3 66 -> 51, 512x512x320 300 -> 222, 171x203x117
// Neumann 38 -> 31 (6 blocks of 128 threads per SM; unlimited and 8 measured slower).
template <typename T, int NI, bool NEU, typename IX = long long>
__device__ __forceinline__ void rb_residual_vec_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ U, const T* __restrict__ B, const Dims& d, const GsCoef<T>& c, double* part, int want_beff, int ni)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    constexpr int lo = NEU ? 0 : 1;
    int g, j;
    const int hz = d.hz();
    flat_pair(blockIdx, (unsigned)(hz / W), g, j);
    const int color = blockIdx.z & 1;
    const int ib = (int)(blockIdx.z >> 1) * ni;
    const int i0 = ib < lo ? lo : ib, i1 = min(ib + ni, d.nx - lo);
    const int m0 = g * W;
    double acc = 0, accb = 0;
    if (j >= lo && j < d.ny - lo && i0 < i1) {
        const IX plane = (IX)d.ny * hz;
        const IX npk = plane * d.nx;
        const IX q0 = ((IX)i0 * d.ny + j) * hz + m0;
        const T* po = U + (color ? 0 : npk) + q0;
        const T* pu = U + (color ? npk : 0) + q0;
        const T* pb = B + (color ? npk : 0) + q0;
        const int cy = j == 0 ? 0 : (j == d.ny - 1 ? 2 : 1);
        const bool has_ym = !NEU || cy != 0, has_yp = !NEU || cy != 2;
        int par = (i0 + j + color) & 1;
        VV ymn = VV{}, ypn = VV{}, bn, un;
        T en = T(0);
        auto side = [&](const T* p, int pr) {
            if (has_ym) ymn = *reinterpret_cast<const VV*>(p - hz);
            if (has_yp) ypn = *reinterpret_cast<const VV*>(p + hz);
            const bool e_ok = pr ? m0 + W < hz : m0 >= 1;
            en = e_ok ? p[pr ? W : -1] : T(0);
        };
        auto to_d = [](const VV& v, double (&o)[W]) {
#pragma unroll
            for (int cc = 0; cc < W; ++cc) o[cc] = (double)VT::get(v, cc);
        };
        double xm[W], xc[W], xp[W];
        {
            VV v = VV{};
            if (!NEU || i0 >= 1) v = *reinterpret_cast<const VV*>(po - plane);
            to_d(v, xm);
            to_d(*reinterpret_cast<const VV*>(po), xc);
        }
        side(po, par);
        bn = *reinterpret_cast<const VV*>(pb);
        un = *reinterpret_cast<const VV*>(pu);
#pragma unroll
        for (int t = 0; t < NI; ++t) {
            const int i = i0 + t;
            if (i >= i1) break;
            const VV ym = ymn, yp = ypn, bv = bn, uv = un;
            const double extra = (double)en;
            VV xv = VV{};
            if (!NEU || i + 1 < d.nx) xv = *reinterpret_cast<const VV*>(po + plane);
            if (t + 1 < NI && i + 1 < i1) {
                side(po + plane, par ^ 1);
                pb += plane;
                pu += plane;
                bn = *reinterpret_cast<const VV*>(pb);
                un = *reinterpret_cast<const VV*>(pu);
            }
            to_d(xv, xp);
            const int last = ((d.nz - 1 - par) >> 1) - m0;    // the last cell with k < nz
            const bool last_k = ((d.nz - 1 - par) & 1) == 0;  // ... and whether its k is nz - 1
            const int cx = NEU ? (i == 0 ? 0 : (i == d.nx - 1 ? 2 : 1)) : 1;
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                const bool at0 = cc == 0 && par == 0 && m0 == 0, at1 = last_k && cc == last;
                double sx = xm[cc] + xp[cc];
                double sy = (double)VT::get(ym, cc) + (double)VT::get(yp, cc);
                double zn = par ? (cc + 1 < W ? xc[cc + 1] : extra) : (cc >= 1 ? xc[cc - 1] : extra);
                double zc = xc[cc];
                double diag = c.diagd;
                if (NEU) {
                    // a missing neighbour was read as 0 (past the row: replaced here)
                    if (at1) {
                        if (par) zn = 0;
                        else zc = 0;
                    }
                    if (at0 || at1 || cx != 1 || cy != 1) {
                        const double bcn = c.bcnd[(cx != 1) + (cy != 1) + (at0 || at1)];
                        if (cx != 1) sx += cx == 0 ? -(bcn * c.hx) : bcn * c.hx;
                        if (cy != 1) sy += cy == 0 ? -(bcn * c.hy) : bcn * c.hy;
                        if (at0) zn += -(bcn * c.hz);
                        if (at1) zn += bcn * c.hz;
                        diag = 1.0 / c.dt + (cx == 1 ? 2.0 : 1.0) * c.ihx2d + (cy == 1 ? 2.0 : 1.0) * c.ihy2d +
                               (at0 || at1 ? 1.0 : 2.0) * c.ihz2d;
                    }
                }
                const double b = (double)VT::get(bv, cc);
                double r = sx * c.ihx2d + sy * c.ihy2d + (zc + zn) * c.ihz2d + b - diag * (double)VT::get(uv, cc);
                const bool unknown = cc <= last && (NEU || !(at0 || at1));
                r = unknown ? r : 0.0;
                acc += r * r;
                if (want_beff) accb += unknown ? b * b : 0.0;
            }
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                xm[cc] = xc[cc];
                xc[cc] = xp[cc];
            }
            po += plane;
            par ^= 1;
        }
    }
    if (want_beff) block_sum2_store(acc, accb, part, block_linear_id(blockIdx, gridDim), grid_blocks(gridDim));
    else block_sum_store(acc, part, block_linear_id(blockIdx, gridDim));
}

template <typename T, int NI, bool NEU, typename IX>
__global__ void __launch_bounds__(128, 6) rb_residual_vec_kernel(const T* __restrict__ U, const T* __restrict__ B, Dims d, GsCoef<T> c, double* part, int want_beff, int ni)
{
    rb_residual_vec_body<T, NI, NEU, IX>(blockIdx, gridDim, U, B, d, c, part, want_beff, ni);
}


// cut_phi (rsfe_splitbregman_imp.hxx:320-339) and the tolerance sums of :1832:
// phi holds phiold on entry and the clamped solve result on exit (natural layout);
// u is the solve result (packed or natural); u_out, when given, receives it unclamped.
template <typename T, bool PACKED, int NI>
__device__ __forceinline__ void clamp_tol_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ u, T* phi, T* __restrict__ u_out, Dims d, T a0, T b0, double* part)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i0 = blockIdx.z * NI;
    double s_d = 0, s_o = 0;
    if (k < d.nz && j < d.ny) {
        const int cnt = min(NI, d.nx - i0);
        const long long plane = (long long)d.ny * d.nz;
        const long long pplane = (long long)d.ny * d.hz();
        const long long p0 = d.idx(i0, j, k);
        const long long pq0 = d.pidx(i0, j, k);
        const long long npk = pplane * d.nx;
        // every load of the NI planes before the first store: a store to phi would
        // otherwise hold the next plane's loads back (one memory round trip per plane)
        T uv[NI], ov[NI];
#pragma unroll
        for (int t = 0; t < NI; ++t) {
            if (t < cnt) {
                const long long p = p0 + t * plane;
                uv[t] = PACKED ? u[pq0 + t * pplane + (((i0 + t + j + k) & 1) ? npk : 0)] : u[p];
                ov[t] = phi[p];
            }
        }
#pragma unroll
        for (int t = 0; t < NI; ++t) {
            if (t < cnt) {
                const long long p = p0 + t * plane;
                if (u_out) u_out[p] = uv[t];
                T v = uv[t];
                if (v < a0) v = a0;
                else if (v > b0) v = b0;
                const T old = ov[t];
                phi[p] = v;
                const double df = (double)v - (double)old;
                s_d += df * df;
                s_o += (double)old * (double)old;
            }
        }
    }
    block_sum2_store(s_d, s_o, part, block_linear_id(blockIdx, gridDim), grid_blocks(gridDim));
}

template <typename T, bool PACKED, int NI>
__global__ void __launch_bounds__(256) clamp_tol_kernel(const T* __restrict__ u, T* phi, T* __restrict__ u_out, Dims d, T a0, T b0, double* part)
{
    clamp_tol_body<T, PACKED, NI>(blockIdx, gridDim, u, phi, u_out, d, a0, b0, part);
}

// The Split-Bregman update on the clamped phi (rsfe_splitbregman_imp.hxx:1868-1906),
// per component c: d = grad(phi)_c; b += d; d = shrink(b, g); b -= d; d -= b.
// Thread per (k, j) column marching over NI planes with phi(i-1), phi(i), phi(i+1)
// in registers; j and k neighbours come through L1.
template <typename T, int NI>
__device__ __forceinline__ void bregman_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ phi, T* __restrict__ b3, T* __restrict__ dmb, const T* __restrict__ g, Dims d, HStep<T> hs)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i0 = blockIdx.z * NI;
    if (k >= d.nz || j >= d.ny) return;
    const int cnt = min(NI, d.nx - i0);
    const long long plane = (long long)d.ny * d.nz;
    const long long n = d.n();
    const long long sy = d.nz;
    const long long p0 = d.idx(i0, j, k);
    // Every load of the NI planes is issued before the first store (the stores to b3
    // and dmb would otherwise hold the next plane's loads back): phi along i for planes
    // i0-1 .. i0+NI (and the second one-sided point on an i face), the j and k
    // neighbours of each plane, g and the three components of b.
    T fi[NI + 2], fi2[NI], fjm[NI], fjp[NI], fkm[NI], fkp[NI], gv[NI], bv0[NI][3];
#pragma unroll
    for (int t = 0; t < NI + 2; ++t) {
        const int i = i0 - 1 + t;
        fi[t] = (i >= 0 && i < d.nx && t <= cnt + 1) ? phi[p0 + (long long)(t - 1) * plane] : T(0);
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        if (t >= cnt) break;
        const int i = i0 + t;
        const long long p = p0 + (long long)t * plane;
        fi2[t] = i == 0 ? phi[p + 2 * plane] : (i == d.nx - 1 ? phi[p - 2 * plane] : T(0));
        if (j == 0) {
            fjp[t] = phi[p + sy];
            fjm[t] = phi[p + 2 * sy];
        } else if (j == d.ny - 1) {
            fjm[t] = phi[p - sy];
            fjp[t] = phi[p - 2 * sy];
        } else {
            fjp[t] = phi[p + sy];
            fjm[t] = phi[p - sy];
        }
        if (k == 0) {
            fkp[t] = phi[p + 1];
            fkm[t] = phi[p + 2];
        } else if (k == d.nz - 1) {
            fkm[t] = phi[p - 1];
            fkp[t] = phi[p - 2];
        } else {
            fkp[t] = phi[p + 1];
            fkm[t] = phi[p - 1];
        }
        gv[t] = g[p];
#pragma unroll
        for (int cmp = 0; cmp < 3; ++cmp) bv0[t][cmp] = b3[cmp * n + p];
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        if (t >= cnt) break;
        const int i = i0 + t;
        const long long p = p0 + (long long)t * plane;
        const T fm = fi[t], f0 = fi[t + 1], fp = fi[t + 2];
        T gr[3];
        if (i == 0) gr[0] = over_two_h<0>(T(4) * fp - T(3) * f0 - fi2[t], hs);
        else if (i == d.nx - 1) gr[0] = over_two_h<0>(T(3) * f0 - T(4) * fm + fi2[t], hs);
        else gr[0] = over_two_h<0>(fp - fm, hs);
        // j == 0: fjp = phi(j+1), fjm = phi(j+2); j == ny-1: fjm = phi(j-1), fjp = phi(j-2)
        if (j == 0) gr[1] = over_two_h<1>(T(4) * fjp[t] - T(3) * f0 - fjm[t], hs);
        else if (j == d.ny - 1) gr[1] = over_two_h<1>(T(3) * f0 - T(4) * fjm[t] + fjp[t], hs);
        else gr[1] = over_two_h<1>(fjp[t] - fjm[t], hs);
        if (k == 0) gr[2] = over_two_h<2>(T(4) * fkp[t] - T(3) * f0 - fkm[t], hs);
        else if (k == d.nz - 1) gr[2] = over_two_h<2>(T(3) * f0 - T(4) * fkm[t] + fkp[t], hs);
        else gr[2] = over_two_h<2>(fkp[t] - fkm[t], hs);
        const T gg = gv[t];
#pragma unroll
        for (int cmp = 0; cmp < 3; ++cmp) {
            T bv = bv0[t][cmp];
            bv += gr[cmp];
            const T mag = fabs(bv) - gg;
            const T sgn = T((int)(bv > T(0)) - (int)(bv < T(0)));
            const T dn = sgn * ((mag < T(0)) ? T(0) : mag);
            bv -= dn;
            b3[cmp * n + p] = bv;
            dmb[cmp * n + p] = dn - bv;
        }
    }
}

template <typename T, int NI>
__global__ void __launch_bounds__(256) bregman_kernel(const T* __restrict__ phi, T* __restrict__ b3, T* __restrict__ dmb, const T* __restrict__ g, Dims d, HStep<T> hs)
{
    bregman_body<T, NI>(blockIdx, gridDim, phi, b3, dmb, g, d, hs);
}

// ---- vectorised natural-layout kernels (nz a multiple of W = 16/sizeof(T)) ----
// Thread per group of W consecutive k of row j, marching over NI planes of i.

// cut_phi + tolerance sums, reading the solve result from the packed layout: for
// natural k = kb .. kb+W-1 (kb even) the even k sit in the colour array of (i+j)&1 and
// the odd k in the other, both at m = kb/2 .. kb/2 + W/2 - 1. Every read of the NI planes
// is issued before the first store (u_out and phi could alias the reads as far as the
// compiler knows, so a read after a store would wait for it: 197 -> 43 us at 256^3 with
// u_out, 512x512x320 1012 -> 209 us).
template <typename T, bool PACKED, int NI>
__device__ __forceinline__ void clamp_tol_vec_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ u, T* phi, T* __restrict__ u_out, Dims d, T a0, T b0, double* part)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    int g, j;
    flat_pair(blockIdx, (unsigned)(d.nz / W), g, j);
    const int i0 = blockIdx.z * NI;
    const int kb = g * W;
    double s_d = 0, s_o = 0;
    if (kb < d.nz && j < d.ny) {
        const long long plane = (long long)d.ny * d.nz;
        const long long pplane = (long long)d.ny * d.hz();
        const long long npk = pplane * d.nx;
        const int cnt = min(NI, d.nx - i0);
        T* pp = phi + d.idx(i0, j, kb);
        VV uv[NI], old[NI];
#pragma unroll
        for (int t = 0; t < NI; ++t) {
            uv[t] = old[t] = VV{};
            if (t >= cnt) continue;
            old[t] = *reinterpret_cast<const VV*>(pp + t * plane);
            if (PACKED) {
                typedef Vec<T, W / 2> VH;
                const int i = i0 + t;
                const T* q = u + ((long long)i * d.ny + j) * d.hz() + (kb >> 1);
                const int c0 = (i + j) & 1;  // colour of the even k
                const VH ev = *reinterpret_cast<const VH*>(q + (c0 ? npk : 0));
                const VH od = *reinterpret_cast<const VH*>(q + (c0 ? 0 : npk));
#pragma unroll
                for (int h = 0; h < W / 2; ++h) {
                    VT::set(uv[t], 2 * h, ev.v[h]);
                    VT::set(uv[t], 2 * h + 1, od.v[h]);
                }
            } else {
                uv[t] = *reinterpret_cast<const VV*>(u + d.idx(i0 + t, j, kb));
            }
        }
#pragma unroll
        for (int t = 0; t < NI; ++t) {
            if (t >= cnt) break;
            if (u_out) *reinterpret_cast<VV*>(u_out + (pp - phi) + t * plane) = uv[t];
            VV nv;
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                T v = VT::get(uv[t], cc);
                if (v < a0) v = a0;
                else if (v > b0) v = b0;
                VT::set(nv, cc, v);
                const double o = (double)VT::get(old[t], cc);
                const double df = (double)v - o;
                s_d += df * df;
                s_o += o * o;
            }
            *reinterpret_cast<VV*>(pp + t * plane) = nv;
        }
    }
    block_sum2_store(s_d, s_o, part, block_linear_id(blockIdx, gridDim), grid_blocks(gridDim));
}

template <typename T, bool PACKED, int NI>
__global__ void __launch_bounds__(256) clamp_tol_vec_kernel(const T* __restrict__ u, T* phi, T* __restrict__ u_out, Dims d, T a0, T b0, double* part)
{
    clamp_tol_vec_body<T, PACKED, NI>(blockIdx, gridDim, u, phi, u_out, d, a0, b0, part);
}

// Split-Bregman update (see bregman_kernel), vectorised along k; rows on an i or j face
// of the volume take the scalar one-sided stencils.
template <typename T, int NI>
__device__ __forceinline__ void bregman_vec_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ phi, T* __restrict__ b3, T* __restrict__ dmb, const T* __restrict__ g3, Dims d, HStep<T> hs)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    int g, j;
    flat_pair(blockIdx, (unsigned)(d.nz / W), g, j);
    const int i0 = blockIdx.z * NI;
    const int kb = g * W;
    if (kb >= d.nz || j >= d.ny) return;
    const long long plane = (long long)d.ny * d.nz;
    const long long sy = d.nz;
    const long long n = d.n();
    const bool jint = j >= 1 && j <= d.ny - 2;
    const long long p0 = d.idx(i0, j, kb);
    VV f[NI + 2];
#pragma unroll
    for (int t = 0; t < NI + 2; ++t) {
        const int i = i0 - 1 + t;
        if (i >= 0 && i < d.nx) f[t] = *reinterpret_cast<const VV*>(phi + p0 + (long long)(t - 1) * plane);
        else f[t] = VV{};
    }
    // every read of the NI planes is issued before the first store: b3 is read and
    // written, so a read placed after a store could not be moved ahead of it
    VV yms[NI], yps[NI], ggs[NI], bos[NI][3];
    T zlo[NI], zhi[NI];
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        const long long p = p0 + (long long)t * plane;
        yms[t] = yps[t] = ggs[t] = VV{};
        bos[t][0] = bos[t][1] = bos[t][2] = VV{};
        zlo[t] = zhi[t] = T(0);
        if (i < d.nx) {
            if (jint && i >= 1 && i <= d.nx - 2) {
                yms[t] = *reinterpret_cast<const VV*>(phi + p - sy);
                yps[t] = *reinterpret_cast<const VV*>(phi + p + sy);
            }
            if (kb >= 1) zlo[t] = phi[p - 1];
            if (kb + W < d.nz) zhi[t] = phi[p + W];
            ggs[t] = *reinterpret_cast<const VV*>(g3 + p);
#pragma unroll
            for (int cmp = 0; cmp < 3; ++cmp) bos[t][cmp] = *reinterpret_cast<const VV*>(b3 + cmp * n + p);
        }
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        if (i >= d.nx) break;
        const long long p = p0 + (long long)t * plane;
        const bool rowint = jint && i >= 1 && i <= d.nx - 2;
        const VV ym = yms[t], yp = yps[t];
        // phi at k = kb-1 .. kb+W of this row: zz[c + 1] = phi[kb + c]
        T zz[W + 2];
        zz[0] = zlo[t];
#pragma unroll
        for (int c = 0; c < W; ++c) zz[c + 1] = VT::get(f[t + 1], c);
        zz[W + 1] = zhi[t];
        const VV gg = ggs[t];
        VV bo[3], dn[3];
#pragma unroll
        for (int cmp = 0; cmp < 3; ++cmp) bo[cmp] = bos[t][cmp];
#pragma unroll
        for (int cc = 0; cc < W; ++cc) {
            const int k = kb + cc;
            T gr[3];
            if (rowint) {
                // i and j inside: central x and y terms; the z term is central or, on
                // the faces k = 0 and k = nz-1, grad_term's one-sided difference,
                // evaluated with the same operations without a branch
                gr[0] = over_two_h<0>(VT::get(f[t + 2], cc) - VT::get(f[t], cc), hs);
                gr[1] = over_two_h<1>(VT::get(yp, cc) - VT::get(ym, cc), hs);
                T tz = over_two_h<2>(zz[cc + 2] - zz[cc], hs);
                if (cc == 0) {
                    const T lo = over_two_h<2>(T(4) * zz[cc + 2] - T(3) * zz[cc + 1] - zz[cc + 3], hs);
                    tz = k == 0 ? lo : tz;
                }
                if (cc == W - 1) {
                    const T hi = over_two_h<2>(T(3) * zz[cc + 1] - T(4) * zz[cc] + zz[cc - 1], hs);
                    tz = k == d.nz - 1 ? hi : tz;
                }
                gr[2] = tz;
            } else {
                const long long pc = p + cc;
                gr[0] = grad_term<0>(phi, pc, plane, i, d.nx, hs);
                gr[1] = grad_term<1>(phi, pc, sy, j, d.ny, hs);
                gr[2] = grad_term<2>(phi, pc, 1, k, d.nz, hs);
            }
            const T gv = VT::get(gg, cc);
#pragma unroll
            for (int cmp = 0; cmp < 3; ++cmp) {
                T bv = VT::get(bo[cmp], cc);
                bv += gr[cmp];
                const T mag = fabs(bv) - gv;
                const T sgn = T((int)(bv > T(0)) - (int)(bv < T(0)));
                const T dd = sgn * ((mag < T(0)) ? T(0) : mag);
                bv -= dd;
                VT::set(bo[cmp], cc, bv);
                VT::set(dn[cmp], cc, dd - bv);
            }
        }
#pragma unroll
        for (int cmp = 0; cmp < 3; ++cmp) {
            *reinterpret_cast<VV*>(b3 + cmp * n + p) = bo[cmp];
            *reinterpret_cast<VV*>(dmb + cmp * n + p) = dn[cmp];
        }
    }
}

template <typename T, int NI>
__global__ void __launch_bounds__(256) bregman_vec_kernel(const T* __restrict__ phi, T* __restrict__ b3, T* __restrict__ dmb, const T* __restrict__ g3, Dims d, HStep<T> hs)
{
    bregman_vec_body<T, NI>(blockIdx, gridDim, phi, b3, dmb, g3, d, hs);
}

// im3d::div vectorised along k (see div_point); rows on an i or j face of the volume
// take the scalar rule with the reference's quirks.
template <typename T, int NI>
__device__ __forceinline__ void div_vec_body(const uint3 blockIdx, const dim3 gridDim, const T* __restrict__ v, T* __restrict__ out, Dims d, HStep<T> hs)
{
    typedef V16<T> VT;
    typedef typename VT::type VV;
    constexpr int W = VT::W;
    int g, j;
    flat_pair(blockIdx, (unsigned)(d.nz / W), g, j);
    const int i0 = blockIdx.z * NI;
    const int kb = g * W;
    if (kb >= d.nz || j >= d.ny) return;
    const long long plane = (long long)d.ny * d.nz;
    const long long sy = d.nz;
    const long long n = d.n();
    const T* f0 = v;
    const T* f1 = v + n;
    const T* f2 = v + 2 * n;
    const bool jint = j >= 1 && j <= d.ny - 2;
    const long long p0 = d.idx(i0, j, kb);
    VV x[NI + 2];
#pragma unroll
    for (int t = 0; t < NI + 2; ++t) {
        const int i = i0 - 1 + t;
        if (i >= 0 && i < d.nx) x[t] = *reinterpret_cast<const VV*>(f0 + p0 + (long long)(t - 1) * plane);
        else x[t] = VV{};
    }
#pragma unroll
    for (int t = 0; t < NI; ++t) {
        const int i = i0 + t;
        if (i >= d.nx) break;
        const long long p = p0 + (long long)t * plane;
        const bool rowint = jint && i >= 1 && i <= d.nx - 2;
        VV o;
        if (rowint) {
            const VV ym = *reinterpret_cast<const VV*>(f1 + p - sy);
            const VV yp = *reinterpret_cast<const VV*>(f1 + p + sy);
            const VV zc = *reinterpret_cast<const VV*>(f2 + p);
            // f2 at k = kb-1 .. kb+W: zz[c + 1] = f2[kb + c]
            T zz[W + 2];
            zz[0] = kb >= 1 ? f2[p - 1] : T(0);
#pragma unroll
            for (int c = 0; c < W; ++c) zz[c + 1] = VT::get(zc, c);
            zz[W + 1] = kb + W < d.nz ? f2[p + W] : T(0);
            // i and j inside: div_point's x and y terms are central, and its z term is
            // central or, on the faces k = 0 and k = nz-1, grad_term's one-sided
            // difference; evaluated here with the same operations, without a branch
#pragma unroll
            for (int cc = 0; cc < W; ++cc) {
                const int k = kb + cc;
                const T tx = over_two_h<0>(VT::get(x[t + 2], cc) - VT::get(x[t], cc), hs);
                const T ty = over_two_h<1>(VT::get(yp, cc) - VT::get(ym, cc), hs);
                T tz = over_two_h<2>(zz[cc + 2] - zz[cc], hs);
                if (cc == 0) {
                    const T lo = over_two_h<2>(T(4) * zz[cc + 2] - T(3) * zz[cc + 1] - zz[cc + 3], hs);
                    tz = k == 0 ? lo : tz;
                }
                if (cc == W - 1) {
                    const T hi = over_two_h<2>(T(3) * zz[cc + 1] - T(4) * zz[cc] + zz[cc - 1], hs);
                    tz = k == d.nz - 1 ? hi : tz;
                }
                VT::set(o, cc, tx + ty + tz);
            }
        } else {
#pragma unroll
            for (int cc = 0; cc < W; ++cc) VT::set(o, cc, div_point(f0, f1, f2, d, i, j, kb + cc, hs));
        }
        *reinterpret_cast<VV*>(out + p) = o;
    }
}

template <typename T, int NI>
__global__ void __launch_bounds__(256) div_vec_kernel(const T* __restrict__ v, T* __restrict__ out, Dims d, HStep<T> hs)
{
    div_vec_body<T, NI>(blockIdx, gridDim, v, out, d, hs);
}

// sum (a - b)^2 and sum b^2 over n elements (relative change of a sweep)
template <typename T>
__global__ void diff_sums_kernel(const T* __restrict__ a, const T* __restrict__ b, long long n,
                                 double* part)
{
    double sd = 0, sb = 0;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const double x = (double)a[q] - (double)b[q];
        sd += x * x;
        sb += (double)b[q] * (double)b[q];
    }
    block_sum2_store(sd, sb, part, block_linear_id(blockIdx, gridDim), grid_blocks(gridDim));
}

// natural -> packed copy of a volume (both colours), and back
template <typename T>
__global__ void pack_kernel(const T* __restrict__ src, T* __restrict__ dst, Dims d)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    dst[d.pidx(i, j, k) + (((i + j + k) & 1) ? d.npk() : 0)] = src[d.idx(i, j, k)];
}

template <typename T>
__global__ void unpack_kernel(const T* __restrict__ src, T* __restrict__ dst, Dims d)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    dst[d.idx(i, j, k)] = src[d.pidx(i, j, k) + (((i + j + k) & 1) ? d.npk() : 0)];
}

// packed b_eff = b + u/dt (u packed), with sum b_eff^2; Dirichlet faces of u := bc
template <typename T>
__global__ void make_beff_kernel(const T* __restrict__ b, T* __restrict__ U, T* __restrict__ Beff,
                                 Dims d, T inv_dt, T bc, int dirichlet, double* part)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    double acc = 0;
    if (k < d.nz && j < d.ny) {
        const long long pq = d.pidx(i, j, k) + (((i + j + k) & 1) ? d.npk() : 0);
        const bool face = i == 0 || j == 0 || k == 0 || i == d.nx - 1 || j == d.ny - 1 ||
                          k == d.nz - 1;
        T u = U[pq];
        if (dirichlet && face) {
            u = bc;
            U[pq] = u;
        }
        const T e = b[d.idx(i, j, k)] + u * inv_dt;
        Beff[pq] = e;
        if (!(dirichlet && face)) acc = (double)e * (double)e;
    }
    if (part) block_sum_store(acc, part, block_linear_id(blockIdx, gridDim));
}


// ------------------------------------------------------------------ utilities
// min / max of a volume as order-preserving unsigned keys (umax[0] = max, umax[1] = max of -x)
__device__ __forceinline__ unsigned long long order_key(double x)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// the same order on the bits of a float or double themselves (NaN included): its key is the
// order_key of the value's double up to the width
template <typename T>
struct KeyOf;
template <>
struct KeyOf<float> {
    typedef unsigned int type;
    static __device__ __forceinline__ type key(float x)
    {
        const unsigned int b = __float_as_uint(x);
        return (b >> 31) ? ~b : (b | 0x80000000u);
    }
    static __device__ __forceinline__ float value(type k)
    {
        return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
    }
};
template <>
struct KeyOf<double> {
    typedef unsigned long long type;
    static __device__ __forceinline__ type key(double x) { return order_key(x); }
    static __device__ __forceinline__ double value(type k)
    {
        return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
    }
};

// umax[0] = order key of the maximum, umax[1] = of minus the minimum, umax[3] raised by a NaN
// or Inf. Bound by the read of the volume: integer keys of the value's own width, eight values
// per thread and round (FP64 keys of every value took 40 us for 12.6 M floats, now 10). One pair
// of atomics per block: one per warp, 38 thousand on one address, took half of 38 us for
// 12.6 M floats out of cache, now 16.
template <typename T>
__global__ void __launch_bounds__(256) minmax_kernel(const T* __restrict__ p, long long n, unsigned long long* umax)
{
    typedef typename KeyOf<T>::type K;
    K mx = 0, mn = ~K(0);
    bool bad = false;
    const long long step = (long long)gridDim.x * blockDim.x;
    long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    auto take = [&](T v) {
        bad |= !isfinite(v);
        const K k = KeyOf<T>::key(v);
        mx = k > mx ? k : mx;
        mn = k < mn ? k : mn;
    };
    constexpr int U = 8;
    for (; q < n; q += U * step) {
        T v[U];
#pragma unroll
        for (int e = 0; e < U; ++e) v[e] = ld_g(p + min(q + e * step, n - 1));
#pragma unroll
        for (int e = 0; e < U; ++e) take(v[e]);
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicMax(umax + 3, 1ull);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const K a = __shfl_xor_sync(0xffffffffu, mx, o), b = __shfl_xor_sync(0xffffffffu, mn, o);
        mx = a > mx ? a : mx;
        mn = b < mn ? b : mn;
    }
    __shared__ K smx[8], smn[8];
    if ((threadIdx.x & 31) == 0) {
        smx[threadIdx.x >> 5] = mx;
        smn[threadIdx.x >> 5] = mn;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
        mx = smx[w] > mx ? smx[w] : mx;
        mn = smn[w] < mn ? smn[w] : mn;
    }
    // (a block that saw no value keeps the neutral keys and adds nothing)
    if (mn <= mx) {
        atomicMax(umax + 0, order_key((double)KeyOf<T>::value(mx)));
        atomicMax(umax + 1, order_key(-(double)KeyOf<T>::value(mn)));
    }
}

// ---- connected component (image3d<T>::connected_component, image3d_imp.hxx:1694-2120) ----
// One bit per cell, 32 cells along the contiguous axis per word, a row of `words` words per
// (a, b): `white` (the black-and-white image: img >= pivot, or img < pivot in the negative
// image) and `comp` (in the component). A volume is rows a = i, b = j of nz cells; a 2-D image
// (nz == 1) is one plane a = 0 of rows b = i of ny cells, whose plane index restricts nothing.
struct CcDims {
    int na, nb, nk, words;
    int plane_rule;  // 1: cells with a = 0 or na - 1 do not spread
    __host__ __device__ long long row(int a, int b) const { return (long long)a * nb + b; }
};

// Row and word of the row of word w; consecutive words are visited with one division.
struct CcWord {
    long long row;
    int k;
    __device__ __forceinline__ CcWord(const CcDims& d, long long w, long long total)
    {
        row = total <= 0x7fffffffLL ? (long long)((unsigned)w / (unsigned)d.words) : w / d.words;
        k = (int)(w - row * d.words);
    }
    __device__ __forceinline__ void next(const CcDims& d)
    {
        if (++k == d.words) {
            k = 0;
            ++row;
        }
    }
};

// im_to_black_and_white (image3d_imp.hxx:1592-1623) and the initial component: the
// cells where init != 0 and white (init != NULL), else only cell `seed` (>= 0). A warp turns
// 4 words of cells into bits: 39 us for 12.6 M floats out of cache with a division per word,
// now 32 (8 words at a time: 34).
template <typename T>
__global__ void __launch_bounds__(256) cc_init_kernel(const T* __restrict__ img, const T* __restrict__ init,
                                                      unsigned* __restrict__ white, unsigned* __restrict__ comp,
                                                      CcDims d, T pivot, int negative, long long seed)
{
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    const long long total = (long long)d.na * d.nb * d.words;
    for (long long w0 = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * U; w0 < total;
         w0 += (long long)gridDim.x * (blockDim.x >> 5) * U) {
        T v[U], in[U];
        bool ok[U];
        long long cell[U];
        CcWord at(d, w0, total);
#pragma unroll
        for (int u = 0; u < U; ++u, at.next(d)) {
            const int k = at.k * 32 + lane;
            ok[u] = w0 + u < total && k < d.nk;
            cell[u] = at.row * d.nk + k;
            v[u] = ok[u] ? ld_g(img + cell[u]) : T(0);
            in[u] = ok[u] && init ? ld_g(init + cell[u]) : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool below = v[u] < pivot;
            const bool wh = ok[u] && (negative ? below : !below);
            const bool c = ok[u] && (init ? in[u] != T(0) && wh : cell[u] == seed);
            const unsigned bw = __ballot_sync(0xffffffffu, wh), bc = __ballot_sync(0xffffffffu, c);
            if (lane == 0 && w0 + u < total) {
                white[w0 + u] = bw;
                comp[w0 + u] = bc;
            }
        }
    }
}

// One growth pass over tiles of kCcW words (k) x kCcB x kCcA rows, in place. A thread owns a
// word; the tile and its one-word, one-row halo hold the spreading cells (in the component and
// off the volume's faces) in shared memory. A round adds the white cells next to a spreading
// one (6 face neighbours, 26 with FULL) and fills each word's runs of white spreading cells
// from the cells in it (a parallel-prefix fill), until the tile is at its fixed point; then
// the words go back and *changed is raised if the tile grew. Growth only turns bits on, a tile
// writes its own words only, and a halo word read while its tile grows is an older state of it:
// passes repeated until none of them grows reach the reference's fixed point whatever the
// order. (A byte per cell, one cell per thread and round took 72 us per pass at 256 x 256 x
// 192 and needed about twice the passes.)
constexpr int kCcW = 2, kCcB = 16, kCcA = 16;
template <bool FULL>
__global__ void __launch_bounds__(kCcW* kCcB* kCcA) cc_grow_kernel(const unsigned* __restrict__ white, unsigned* comp,
                                                                   CcDims d, unsigned long long* changed,
                                                                   unsigned long long bit)
{
    constexpr int SW = kCcW + 2, SB = kCcB + 2, SA = kCcA + 2, NT = kCcW * kCcB * kCcA;
    __shared__ unsigned tile[SA * SB * SW];
    volatile unsigned* t = tile;
    const int w0 = blockIdx.x * kCcW, b0 = blockIdx.y * kCcB, a0 = blockIdx.z * kCcA;
    const int tid = threadIdx.x;
    // cells of word w that spread, by the rule along k
    auto kmask = [&](int w) {
        unsigned m = 0xffffffffu;
        if (w == 0) m &= ~1u;
        const int last = d.nk - 1 - 32 * w;  // bit of the face cell k = nk - 1, if in this word
        if (last <= 31) m &= last > 0 ? (1u << last) - 1u : 0u;
        return m;
    };
    auto row_spreads = [&](int a, int b) {
        return (!d.plane_rule || (a >= 1 && a <= d.na - 2)) && b >= 1 && b <= d.nb - 2;
    };
    unsigned seen = 0;
    for (int e = tid; e < SA * SB * SW; e += NT) {
        const int la = e / (SB * SW), r = e - la * SB * SW, lb = r / SW, lw = r - lb * SW;
        const int a = a0 - 1 + la, b = b0 - 1 + lb, w = w0 - 1 + lw;
        unsigned v = 0;
        if (a >= 0 && a < d.na && b >= 0 && b < d.nb && w >= 0 && w < d.words && row_spreads(a, b))
            v = __ldcg(comp + d.row(a, b) * d.words + w) & kmask(w);
        t[e] = v;
        seen |= v;
    }
    if (!__syncthreads_or(seen != 0)) return;  // nothing here or next to it spreads
    const int lw = tid % kCcW + 1, lb = tid / kCcW % kCcB + 1, la = tid / (kCcW * kCcB) + 1;
    const int w = w0 + lw - 1, b = b0 + lb - 1, a = a0 + la - 1;
    const bool live = w < d.words && b < d.nb && a < d.na;
    const long long q = live ? d.row(a, b) * d.words + w : 0;
    const unsigned W = live ? __ldg(white + q) : 0u;
    const unsigned S = live && row_spreads(a, b) ? kmask(w) : 0u;
    const unsigned P = W & S;
    const int at = (la * SB + lb) * SW + lw;
    unsigned c = live ? __ldcg(comp + q) : 0u;
    const unsigned start = c;
    bool step;
    do {
        unsigned nb = 0;
#pragma unroll
        for (int da = -1; da <= 1; ++da)
#pragma unroll
            for (int db = -1; db <= 1; ++db) {
                if (!FULL && da != 0 && db != 0) continue;
                const int o = at + (da * SB + db) * SW;
                const unsigned v = t[o];
                nb |= v;
                // the cells beside it along k: its own row's, and with FULL every row's
                if (FULL || (da == 0 && db == 0)) nb |= (v << 1) | (v >> 1) | (t[o - 1] >> 31) | (t[o + 1] << 31);
            }
        unsigned n = c | (W & nb);
        // runs of white spreading cells, from the cells in them, both ways
        unsigned up = n & S, dn = up, pu = P, pd = P;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            up |= pu & (up << s);
            dn |= pd & (dn >> s);
            pu &= pu << s;
            pd &= pd >> s;
        }
        n |= up | dn;
        step = n != c;
        c = n;
        if (step) t[at] = c & S;
    } while (__syncthreads_or(step));
    if (c != start) comp[q] = c;
    if (__syncthreads_or(c != start) && tid == 0) atomicOr(changed, bit);
}

// The result: the component as 0 / 1, or with binary == 0 cc_not_binary_output
// (image3d_imp.hxx:1801-1817): (res + [img < pivot]) * (img - mn) + mn.
template <typename T>
__global__ void __launch_bounds__(256) cc_output_kernel(const unsigned* __restrict__ comp, const T* img, T* res, CcDims d,
                                                        int binary, T mn, T pivot)
{
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    const long long total = (long long)d.na * d.nb * d.words;
    for (long long w0 = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * U; w0 < total;
         w0 += (long long)gridDim.x * (blockDim.x >> 5) * U) {
        CcWord at(d, w0, total);
#pragma unroll
        for (int u = 0; u < U; ++u, at.next(d)) {
            const long long w = w0 + u;
            const int k = at.k * 32 + lane;
            if (w >= total || k >= d.nk) continue;
            const long long q = at.row * d.nk + k;
            T v = (T)(comp[w] >> lane & 1u);
            if (!binary) {
                const T x = img[q];
                v += (T)(x < pivot ? 1 : 0);
                v *= x - mn;
                v += mn;
            }
            res[q] = v;
        }
    }
}

// change_range_of_intensity(max, min) (image3d_imp.hxx:1628-1636) once the minimum
// mn and the shifted maximum are known: x -= mn; x /= s; x += lo
template <typename T>
__global__ void affine_kernel(T* p, long long n, T mn, T s, T lo)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        T x = p[q];
        x -= mn;
        x /= s;
        x += lo;
        p[q] = x;
    }
}

// initialize_phi_with_cube (rsfe_splitbregman_imp.hxx:48-95): a0 outside the box
// [ix, fx) x [iy, fy) x [iz, fz), b0 inside
template <typename T>
__global__ void cube_kernel(T* p, Dims d, int ix, int iy, int iz, int fx, int fy, int fz, T a0,
                            T b0)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const bool in = i >= ix && i < fx && j >= iy && j < fy && k >= iz && k < fz;
    p[d.idx(i, j, k)] = in ? b0 : a0;
}

// ---- learned warm start: fields of one Poisson solve to and from the network ----
// Packed cell of natural (i, j, k): its colour's array at d.pidx(i, j, k).
__device__ __forceinline__ long long packed_at(const Dims& d, int i, int j, int k)
{
    return d.pidx(i, j, k) + (((i + j + k) & 1) ? d.npk() : 0);
}

// The network's inputs, four FP32 volumes x[f][n] (natural layout): the forcing term
// rhs = b_eff - u_in / dt, the previous solve's u, div(d - b) and phi.
static __global__ void ws_fields_kernel(const float* __restrict__ bpk, const float* __restrict__ upk,
                                 const float* __restrict__ prevu, const float* __restrict__ divdb,
                                 const float* __restrict__ phi, Dims d, float inv_dt, float* __restrict__ x)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long v = d.idx(i, j, k), pv = packed_at(d, i, j, k), n = d.n();
    x[v] = bpk[pv] - upk[pv] * inv_dt;
    x[n + v] = prevu[v];
    x[2 * n + v] = divdb[v];
    x[3 * n + v] = phi[v];
}

// u_in += the network's correction y on the cells the solve updates (all cells with
// Neumann conditions, the interior with Dirichlet ones, whose faces keep their value).
static __global__ void ws_apply_kernel(float* __restrict__ upk, const float* __restrict__ y, Dims d, int dirichlet)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    if (dirichlet && (i == 0 || j == 0 || k == 0 || i == d.nx - 1 || j == d.ny - 1 || k == d.nz - 1)) return;
    upk[packed_at(d, i, j, k)] += y[d.idx(i, j, k)];
}

// The correction the solve made, natural layout: t = u_solved - u_in.
static __global__ void ws_target_kernel(const float* __restrict__ upk, const float* __restrict__ upk0, Dims d,
                                 float* __restrict__ t)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= d.nz || j >= d.ny) return;
    const long long pv = packed_at(d, i, j, k);
    t[d.idx(i, j, k)] = upk[pv] - upk0[pv];
}

}  // namespace im3d
