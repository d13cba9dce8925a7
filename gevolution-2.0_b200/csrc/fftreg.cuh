// fftreg.cuh -- two-step register FFTs of the pencil passes.
//
// A line of length L = R1 R2 is transformed by R2 threads in two steps with
// one exchange through shared memory (Cooley-Tukey with n = j + R2 r and
// k = q + R1 p):
//   step 1  thread j holds x[j + R2 r], r < R1: R1-point DFT over r in
//           registers, times exp(S 2 pi i j q / L), to row q of the exchange
//           buffer at position j;
//   step 2  row q (threads take the rows q = u, u + R2, ...) holds R2 values:
//           R2-point DFT over j gives X[q + R1 p], p < R2, in natural order.
// The inverse runs the same two steps backwards (step 2 over p first), so a
// pass over one component that transforms, solves point by point and transforms
// back touches shared memory four times per value and needs two block barriers:
// the values of row q belong to one thread from the exchange to the exchange
// back.  (Several components meet in shared memory for their solve: four more
// accesses and two more barriers.)  Passes bound by shared memory when they run
// radix-8 steps through it (two accesses per step and direction) become bound
// by their global traffic, as long as the 2 R1 or 2 R2 values of a thread leave
// registers for enough warps.
//
// Rows of the exchange buffer have the pitch (R2 + 1) * T (T lines side by
// side, line index fastest): step 1 writes along a row, step 2 reads rows a
// pitch apart, and with the odd number of T-groups in a pitch neither
// conflicts in the banks.
#pragma once

#include <utility>

#include "common.cuh"
#include "fft.cuh"

namespace gev {

// ---- compile-time roots of unity: cos(2 pi k / 96) from the first quadrant ----
// (32 and 24 both divide 96; every composite radix below divides it)
__host__ __device__ constexpr double root_quadrant(int k)   // cos(2 pi k / 96), 0 <= k <= 24
{
    constexpr double c[25] = {
        1.0, 0.99785892323860350, 0.99144486137381038, 0.98078528040323043, 0.96592582628906831, 0.94693012949510569,
        0.92387953251128674, 0.89687274153268836, 0.86602540378443871, 0.83146961230254524, 0.79335334029123517,
        0.75183980747897738, 0.70710678118654757, 0.65934581510006895, 0.60876142900872066, 0.55557023301960218,
        0.5, 0.44228869021900125, 0.38268343236508978, 0.32143946530316153, 0.25881904510252074, 0.19509032201612825,
        0.13052619222005157, 0.065403129230143062, 0.0};
    return c[k];
}
__host__ __device__ constexpr double root_cos(int k)   // cos(2 pi k / 96), any k >= 0
{
    k %= 96;
    if (k > 48) k = 96 - k;
    return k <= 24 ? root_quadrant(k) : -root_quadrant(48 - k);
}
__host__ __device__ constexpr double root_sin(int k) { return root_cos(k + 72); }

// a * exp(S 2 pi i K / R), R a divisor of 96.
// EXACT: in FP32, radices of 16 and 32 carry the rounding errors of the root's
// two constants along, four operations more: such a radix multiplies by one
// root per value more than the radix-8 steps of a Stockham transform, and
// without this the FP32 transforms were the less exact ones (forward and back
// of white noise against 64 bits, x 1e-7; Stockham / two-step / EXACT: 128^3
// 2.49 / 2.50 / 2.36, 256^3 2.71 / 2.77 / 2.43, 384^3 3.05 / 3.13 / 2.87, 512^3
// 2.86 / 2.96 / 2.63, 768^3 3.14 / 3.28 / 3.05).  Time: a phi solve at 384^3 909
// -> 917 us, none that shows at the other sizes; with the radices of 12 and 24
// too it would be 15 us more.  Not for vector fields: what is left of B_i after
// its longitudinal part is gone carries the FP32 rounding of the z pass's last
// sums in a few long modes, ten times all other errors of its transforms (256^3
// at z = 100: 8.4e-5 / 8.6e-5 / 8.5e-5), and its z pass would take 2 % longer.
template <int R, int K, int S, bool EXACT, class C> __device__ __forceinline__ C mul_root(C a)
{
    static_assert(96 % R == 0, "roots are tabulated for divisors of 96");
    using F = decltype(a.x);
    constexpr int k = (K % R) * (96 / R);
    C o;
    if constexpr (k == 0) return a;
    else if constexpr (k == 24) return cmul_si<S>(a);
    else if constexpr (k == 48) { o.x = -a.x; o.y = -a.y; return o; }
    else if constexpr (k == 72) return cmul_si<-S>(a);
    else if constexpr (k == 12 || k == 36 || k == 60 || k == 84) {
        constexpr F r2 = F(0.70710678118654757);
        constexpr int sc = (k == 12 || k == 84) ? 1 : -1, ss = ((k == 12 || k == 36) ? 1 : -1) * S;
        o.x = r2 * (sc * a.x - ss * a.y);
        o.y = r2 * (sc * a.y + ss * a.x);
        return o;
    } else {
        constexpr F c = F(root_cos(k)), s = F(S * root_sin(k));
        if constexpr (EXACT && sizeof(F) == 4 && (R == 16 || R == 32)) {
            constexpr F cl = F(root_cos(k) - (double)c), sl = F(S * root_sin(k) - (double)s);
            o.x = fmaf(a.x, c, fmaf(-a.y, s, a.x * cl - a.y * sl));
            o.y = fmaf(a.y, c, fmaf(a.x, s, a.y * cl + a.x * sl));
        } else {
            o.x = a.x * c - a.y * s;
            o.y = a.y * c + a.x * s;
        }
        return o;
    }
}

template <int V> struct IntC { static constexpr int v = V; };
template <class FN, int... I> __device__ __forceinline__ void static_seq(FN &&f, std::integer_sequence<int, I...>)
{
    (f(IntC<I>{}), ...);
}
template <int N, class FN> __device__ __forceinline__ void static_for(FN &&f)
{
    static_seq(static_cast<FN &&>(f), std::make_integer_sequence<int, N>{});
}

// first factor of a composite in-register radix
template <int R> __host__ __device__ constexpr int radix_a() { return R == 16 ? 4 : (R == 32 ? 4 : (R == 24 ? 3 : (R == 12 ? 3 : (R == 6 ? 2 : 1)))); }

// R-point DFT in registers, natural order in and out, exponent sign S
template <int R, int S, bool EXACT, class C> __device__ __forceinline__ void dft_reg(C (&v)[R])
{
    if constexpr (R == 1) {
        return;
    } else if constexpr (R == 2 || R == 3 || R == 4 || R == 8) {
        dftR<R, S>(v);
    } else {
        constexpr int A = radix_a<R>(), B = R / A;
        static_assert(A > 1 && A * B == R, "unsupported radix");
        C o[R];
        static_for<B>([&](auto bc) {
            constexpr int b = decltype(bc)::v;
            C t[A];
#pragma unroll
            for (int a = 0; a < A; a++) t[a] = v[b + B * a];
            dftR<A, S>(t);
            static_for<A>([&](auto ac) {
                constexpr int a = decltype(ac)::v;
                v[b + B * a] = mul_root<R, b * a, S, EXACT>(t[a]);
            });
        });
#pragma unroll
        for (int a = 0; a < A; a++) {
            C t[B];
#pragma unroll
            for (int b = 0; b < B; b++) t[b] = v[b + B * a];
            dftR<B, S>(t);
#pragma unroll
            for (int b = 0; b < B; b++) o[a + A * b] = t[b];
        }
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = o[r];
    }
}

// R1 and R2 of a line length: R2 threads per line, R1 values per thread in step 1
template <int L> struct RegPlan;
#define GEV_RPLAN(LV, A, B)                                     \
    template <> struct RegPlan<LV> {                            \
        static constexpr int R1 = A, R2 = B;                    \
        static_assert(A * B == LV, "plan");                     \
    };
GEV_RPLAN(8, 4, 2)
GEV_RPLAN(16, 4, 4)
GEV_RPLAN(32, 8, 4)
GEV_RPLAN(64, 8, 8)
GEV_RPLAN(128, 16, 8)
GEV_RPLAN(192, 16, 12)
GEV_RPLAN(256, 16, 16)
GEV_RPLAN(384, 24, 16)
GEV_RPLAN(512, 32, 16)
GEV_RPLAN(768, 32, 24)
#undef GEV_RPLAN

// one complex value global -> shared, asynchronously; zero when !live (src
// must be a valid address all the same)
template <class C> __device__ __forceinline__ void copy_async(C *dst, const C *src, bool live)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = live ? (int)sizeof(C) : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(sizeof(C)), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest K groups of this thread's copies have arrived
template <int K> __device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }

// exchange buffer of T lines of length L, in complex values
template <int L, int T> __host__ __device__ constexpr int exch_size() { return RegPlan<L>::R1 * (RegPlan<L>::R2 + 1) * T; }

// step 1, forward or the end of an inverse: values of thread j to / from the
// exchange column at position j (buf already offset to line t)
template <int L, int S, bool EXACT, int T, class C>
__device__ __forceinline__ void step1_store(C (&v)[RegPlan<L>::R1], C *buf, int j, const C *__restrict__ tw)
{
    constexpr int R1 = RegPlan<L>::R1, R2 = RegPlan<L>::R2;
    dft_reg<R1, S, EXACT>(v);
#pragma unroll
    for (int q = 0; q < R1; q++) {
        if (q > 0) {
            C w = __ldg(tw + q * j);
            if constexpr (S > 0) w.y = -w.y;
            v[q] = cmul(v[q], w);
        }
        buf[(q * (R2 + 1) + j) * T] = v[q];
    }
}

template <int L, int S, bool EXACT, int T, class C>
__device__ __forceinline__ void step1_load(C (&v)[RegPlan<L>::R1], const C *buf, int j)
{
    constexpr int R1 = RegPlan<L>::R1, R2 = RegPlan<L>::R2;
#pragma unroll
    for (int q = 0; q < R1; q++) v[q] = buf[(q * (R2 + 1) + j) * T];
    dft_reg<R1, S, EXACT>(v);
}

// step 2: row q of the exchange buffer, transformed over its R2 values
template <int L, int S, bool EXACT, int T, class C>
__device__ __forceinline__ void step2_load(C (&v)[RegPlan<L>::R2], const C *buf, int q)
{
    constexpr int R2 = RegPlan<L>::R2;
#pragma unroll
    for (int j = 0; j < R2; j++) v[j] = buf[(q * (R2 + 1) + j) * T];
    dft_reg<R2, S, EXACT>(v);
}

// inverse of step 2: transform the row over p, twiddle, back to the buffer
template <int L, int S, bool EXACT, int T, class C>
__device__ __forceinline__ void step2_store(C (&v)[RegPlan<L>::R2], C *buf, int q, const C *__restrict__ tw)
{
    constexpr int R2 = RegPlan<L>::R2;
    dft_reg<R2, S, EXACT>(v);
#pragma unroll
    for (int j = 0; j < R2; j++) {
        if (j > 0) {
            C w = __ldg(tw + q * j);
            if constexpr (S > 0) w.y = -w.y;
            v[j] = cmul(v[j], w);
        }
        buf[(q * (R2 + 1) + j) * T] = v[j];
    }
}

}  // namespace gev
