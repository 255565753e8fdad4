// bk_ops.cu -- launchers of the BK1 / BK3 / BK5 kernels for ONE arithmetic
// engine, chosen at compile time by BK_ENGINE_TU (0 dfma, 1 float-float,
// 2 fp32, 3 mixed): the build compiles this file once per engine so that the
// translation units build in parallel.  Run-time order p -> compile-time Q
// (the role of bk::with_order, include/bk_common.h:148-178).
#include <type_traits>

#include <cuda_runtime.h>

#include "bk_internal.h"
#include "bk5_col.cuh"
#include "bk_adjoint.cuh"
#include "bk_kernels.cuh"

#ifndef BK_ENGINE_TU
#error "BK_ENGINE_TU must be 0 (dfma), 1 (ff), 2 (fp32) or 3 (mixed)"
#endif
// BK_OP_TU selects the operator of this translation unit: 1 BK1, 3 BK3,
// 5 BK5 sweep kernel and 6 BK5 column kernel (one G layout each,
// BK_LAYOUT_TU), 7 the BK3 adjoint and the BK5 dispatch.
#ifndef BK_OP_TU
#error "BK_OP_TU must be 1, 3, 5, 6 or 7"
#endif

namespace bkg {

#if BK_ENGINE_TU == 0
using Eng = EngDfma;
#define BK_SFX dfma
#elif BK_ENGINE_TU == 1
using Eng = EngFF;
#define BK_SFX ff
#elif BK_ENGINE_TU == 2
using Eng = EngF32;
#define BK_SFX f32
#else
using Eng = EngMixed;
#define BK_SFX mixed
#endif

#define BK_CAT2(a, b) a##_##b
#define BK_CAT(a, b) BK_CAT2(a, b)

#ifndef BK_LAYOUT_TU
#define BK_LAYOUT_TU 9
#endif
// A namespace of its own per translation unit: every unit compiles this file,
// and nvcc may give an anonymous namespace the same name in all of them, so
// same-named helpers of different engines or layouts would be merged (or
// clash) at link time.
#define BK_NS3_(a, b, c) tu_##a##_##b##_##c
#define BK_NS3(a, b, c) BK_NS3_(a, b, c)
#define BK_TU_NS BK_NS3(BK_ENGINE_TU, BK_OP_TU, BK_LAYOUT_TU)

namespace BK_TU_NS {

// Elements per block where no measurement says otherwise: about 128 lines per
// sweep (Q^2 lines per element).
constexpr int default_eb(int q) { return (q * q >= 100) ? 1 : ((q * q >= 64) ? 2 : (128 + q * q - 1) / (q * q)); }

// Elements per block of the even-odd kernels, the fastest measured per engine
// and q on GB300 at 2^23..2^26 points per apply, with the batches dealt (Walk;
// shared dynamically, BK3's q = 8 was measured again and moved).  A sweep gives each thread a
// line, so an EB whose EB q^2 lines just fill whole warps leaves no thread
// idle: q = 3: 7 or 14 (63, 126 lines), q = 5: 5 (125), q = 6: 7 (252),
// q = 7: 5 (245).  Where fewer elements per block let more blocks share an
// SM, that wins (from q = 7 the FP32-storage forms, one element).  Times in us
// (previous choice -> this): float-float BK5 q = 3 262 -> 217, q = 5 716 ->
// 597, BK3 q = 3 246 -> 221, q = 5 447 -> 399, BK1 q = 3 203 -> 185, q = 9
// 485 -> 430; FP32 BK5 q = 2 297 -> 250, q = 3 262 -> 244, q = 5 220 -> 197,
// BK3 q = 6 254 -> 234, q = 7 253 -> 235, BK1 q = 3 216 -> 187, q = 7 178 ->
// 162, q = 9 170 -> 145.
constexpr bool eng_is_dfma() { return Eng::kId == BK_ENGINE_DFMA; }
constexpr bool eng_is_ff() { return Eng::kId == BK_ENGINE_FF; }
constexpr int sweep_eb5(int q)
{
    if (eng_is_dfma()) return q <= 3 ? 16 : q == 4 ? 8 : q == 5 ? 6 : q == 6 ? 4 : q == 7 ? 3 : q == 8 ? 2 : 3;
    if (q == 2) return 16;
    if (q == 3) return eng_is_ff() ? 7 : 14;
    if (q <= 6) return q == 4 ? 8 : q == 5 ? 5 : 3;
    return eng_is_ff() && q == 7 ? 4 : 1;
}
constexpr int sweep_eb3(int q)
{
    if (eng_is_dfma())
        return q <= 3 ? 16 : q == 4 ? 8 : q == 5 ? 6 : q == 6 ? 4 : q == 7 ? 3 : q == 8 ? 2 : q == 9 ? 3 : 1;
    if (q <= 4) return q == 3 ? 14 : 8;
    if (eng_is_ff()) return q == 5 ? 10 : q == 6 ? 3 : 1;
    return q == 5 ? 5 : q == 6 ? 7 : 1;
}
// BK1.  At q = 5 the FP32-storage forms also run at EB = 10 (172 -> 166 us at
// E = 500000); 5 keeps the smaller blocks for the small applies
constexpr int sweep_eb1(int q)
{
    if (eng_is_dfma()) return default_eb(q);
    if (eng_is_ff()) return q == 3 ? 14 : q == 8 ? 1 : q == 9 ? 3 : default_eb(q);
    constexpr int t[8] = {14, 8, 5, 7, 5, 1, 1, 1};   // q = 3..10
    return t[q - 3];
}
// the BK3 adjoint (six boxes and two gradients per element)
constexpr int adj_eb(int q)
{
    if (eng_is_dfma()) return default_eb(q) / 2 > 0 ? default_eb(q) / 2 : 1;
    if (eng_is_ff()) return q == 3 ? 7 : q == 4 ? 4 : q == 5 ? 5 : q == 6 ? 3 : 1;
    return q == 3 ? 14 : q == 4 ? 8 : q == 5 ? 5 : q == 6 ? 3 : 1;
}

// The general contractions (matrices without the symmetry): elements per block
// of their own where the tables above, measured with the even-odd ones, lose (us
// at 25 M points with them -> with these: float-float BK3 q = 7 1962 -> 1581,
// FP32 BK1 q = 6 156 -> 147, q = 7 173 -> 151; float-float BK1 q = 9 at 0.06 M
// points 11.6 -> 10.4).
constexpr int gen_eb1(int q)
{
    if (eng_is_ff()) return default_eb(q);
    return q == 6 || q == 7 ? default_eb(q) : sweep_eb1(q);
}
constexpr int gen_eb3(int q) { return eng_is_ff() && q == 7 ? 3 : sweep_eb3(q); }

// Sets the dynamic shared-memory size of a kernel on the current device once
// and returns its resident blocks per SM (0 if it cannot run).  Tag makes the
// cache one per kernel instantiation (kernels of one signature share K).
template <class Cfg, bool EO>
struct EoTag {};

template <class Tag, class K>
int prepare(K kern, int smem, int nt)
{
    static int occ[kMaxDevices] = {0};
    const int dev = current_device();
    if (dev < 0 || dev >= kMaxDevices) return 0;
    if (occ[dev] == 0) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, nt, smem) != cudaSuccess) return 0;
        occ[dev] = n;
    }
    return occ[dev];
}

int grid_for(long long nbatch, int occ)
{
    const long long cap = static_cast<long long>(occ) * sm_count();
    return static_cast<int>(nbatch < cap ? nbatch : cap);
}

// Launches of this many batches per resident block or more walk dynamically
// (Walk<true>, a block per batch in the grid), smaller ones are dealt.  Times
// dealt / dynamic: BK5 p=4 float-float at 2, 4, 8, 16 waves 18.7 / 20.5, 35.1 /
// 37.0, 64.8 / 64.3, 125 / 120 us; BK3 p=5 FP32 at 4, 8, 15 waves 24.8 / 23.2,
// 45.4 / 45.2, 85.7 / 82.1.
// One line for all: float-float loses below it, and FP32 storage, which these
// figures would let share from 4 on, gives up at most a tenth there.
constexpr int kDynWaves = 8;

// One launch of a batch kernel: dealt (sk) or dynamic (dk) by the batches per
// resident block, with `smem` bytes.  EB elements a batch; args: the kernel's.
template <class Tag, bool DYN>
struct WalkTag {};
template <class Cfg, bool EO, int EB, class K, class... Args>
int launch_walk(K sk, K dk, long long E, cudaStream_t s, const Args&... args)
{
    const long long nbatch = (E + EB - 1) / EB;
    const int occ = prepare<WalkTag<EoTag<Cfg, EO>, false>>(sk, Cfg::SMEM, Cfg::NT);
    if (occ <= 0) return BK_ERR_CUDA;
    if (sk != dk && nbatch >= static_cast<long long>(kDynWaves) * occ * sm_count() && nbatch <= 0x7fffffffLL) {
        if (prepare<WalkTag<EoTag<Cfg, EO>, true>>(dk, Cfg::SMEM, Cfg::NT) <= 0) return BK_ERR_CUDA;
        dk<<<static_cast<int>(nbatch), Cfg::NT, Cfg::SMEM, s>>>(args..., dev_ctx());
    } else {
        sk<<<grid_for(nbatch, occ), Cfg::NT, Cfg::SMEM, s>>>(args..., dev_ctx());
    }
    return cudaGetLastError() == cudaSuccess ? BK_OK : BK_ERR_CUDA;
}

// The shapes above were measured on launches of many waves.  One of a few waves
// ends with its fullest SM, so a second shape of fewer elements, or of the
// direction groups (which share an element's lines among three times the threads
// and so are done sooner where an SM has little to do), is kept beside a large
// one, and taken for up to `few` batches of the large shape per SM, and from
// there to kFewPerSm where the elements that the fullest SM has room for times
// the cost of an element are fewer.  cost: of an element in the second shape
// where both fill the chip, in per cent of one in the large shape; 0: no second
// shape.  Both give the same bits.  Measured at 26 sizes of each shape (5e3 to
// 4e6 points) against the large shape alone: float-float BK5 q = 6 0.73 to 0.82
// of its time below 1.3 batches per SM, q = 7 0.57 to 0.9 up to three, BK3 q = 6
// 0.81 below one and 0.82 at 3.7, q = 5 0.94, BK1 q = 9 0.80 to 0.95, adjoint q =
// 5 0.87 to 0.95; FP32 adjoint q = 5 and 6 0.91, BK1 q = 6 and 7 0.91 to 0.99.
struct Few {
    int eb, dpar, few, cost;
};
constexpr int kFewPerSm = 24;
constexpr Few kNoFew{1, 0, 0, 0};
constexpr Few few5(int q)
{
    return !eng_is_ff() ? kNoFew : q == 6 ? Few{4, 2, 1, 102} : q == 7 ? Few{2, 3, 3, 103} : kNoFew;
}
constexpr Few few3(int q)
{
    return !eng_is_ff() ? kNoFew : q == 5 ? Few{8, 0, 0, 110} : q == 6 ? Few{3, 2, 4, 104} : kNoFew;
}
constexpr Few few1(int q)
{
    if (eng_is_dfma()) return kNoFew;
    if (eng_is_ff()) return q == 9 ? Few{2, 0, 0, 110} : kNoFew;
    return q == 6 ? Few{4, 0, 0, 105} : q == 7 ? Few{3, 0, 0, 103} : kNoFew;
}
constexpr Few few_adj(int q)
{
    if (eng_is_dfma()) return kNoFew;
    if (eng_is_ff()) return q == 5 ? Few{3, 0, 0, 102} : kNoFew;
    return q == 5 ? Few{3, 0, 0, 107} : q == 6 ? Few{2, 0, 0, 103} : kNoFew;
}

// Whether the second shape f is taken instead of the large one (eb elements per
// block).
inline bool take_few(long long E, int eb, const Few& f)
{
    const long long sms = sm_count();
    auto batches = [&](int n) { return (E + n - 1) / n; };
    auto room = [&](int n) { return (batches(n) + sms - 1) / sms * n; };   // of the fullest SM
    if (batches(eb) > kFewPerSm * sms) return false;
    return batches(eb) <= f.few * sms || room(f.eb) * f.cost <= room(eb) * 100;
}

#if BK_OP_TU == 5
// One launch of bk5_kernel with the given shape.
// GS: the type G is stored in (the storage type, or ff2 pairs split ahead of
// time for the float-float engine).
template <int Q, int EB, int F, int LAYOUT, bool EO, int DPAR, class GS = typename Eng::S>
int bk5_launch(const P5<typename Eng::C, Q>& prm, long long E, const void* u, const void* G, const void* mass,
               double lambda, void* v, cudaStream_t s)
{
    using Cfg = BK5Cfg<Eng, Q, EB, F, LAYOUT, DPAR>;
    using S = typename Eng::S;
    static_assert(Cfg::SMEM <= 232448, "BK5 block exceeds the shared memory of an SM");
    // dynamic for the even-odd kernels
    return launch_walk<Cfg, EO, EB>(&bk5_kernel<Eng, Q, EB, F, LAYOUT, EO, DPAR, GS, false>,
                                    &bk5_kernel<Eng, Q, EB, F, LAYOUT, EO, DPAR, GS, EO>, E, s, prm, E,
                                    static_cast<const S*>(u), static_cast<const GS*>(G), static_cast<const S*>(mass),
                                    lambda, static_cast<S*>(v));
}

// the largest EB <= EB0 whose block fits an SM's shared memory
template <int Q, int F, int EB0, int DPAR = 0>
constexpr int fit_eb5()
{
    if constexpr (EB0 > 1 && BK5Cfg<Eng, Q, EB0, F, BK_LAYOUT_TU, DPAR>::SMEM > 232448)
        return fit_eb5<Q, F, EB0 - 1, DPAR>();
    else
        return EB0;
}

// The direction-parallel even-odd shape (three thread groups, one direction
// each) for the float-float engine where it measured faster on GB300: q = 8
// (EB 1, one code body for the three directions: 711 us against 910 with one
// thread per line at E = 65536) and q = 9 (EB 3, a body per direction: 939
// against 1010, one shared body 958, at E = 46000).  q = 6 and 7 run one
// thread per line (857 against 869, 875 against 899).
constexpr int sweep_dpar5(int q) { return !eng_is_ff() ? 0 : q == 8 ? 2 : q == 9 ? 1 : 0; }
constexpr int sweep_eb5_dpar(int q) { return q == 9 ? 3 : 1; }

template <int Q>
int bk5_sweep_q(int F, const double* D, long long E, const void* u, const void* G, const void* mass,
                double lambda, void* v, int gform, cudaStream_t s)
{
    constexpr int L = BK_LAYOUT_TU;
    P5<typename Eng::C, Q> prm;
    for (int i = 0; i < Q * Q; ++i) prm.D[i] = Eng::coef(D[i]);
    // the even-odd contractions when D is centro-antisymmetric (GLL points);
    // instantiated for the symmetric 6-factor G only
    const bool eo = (F == 6) && make_eo<typename Eng::C, Q>(D, false, prm.eo, &Eng::coef) &&
                    make_eo<typename Eng::C, Q>(D, true, prm.eot, &Eng::coef);
    if (eo) {
        constexpr int DP = sweep_dpar5(Q);
        constexpr int EB = fit_eb5<Q, 6, DP ? sweep_eb5_dpar(Q) : sweep_eb5(Q), DP>();
        // gs: G as stored, or split ahead of time (the float-float engine)
        auto go = [&](auto gs) {
            using GS = decltype(gs);
            if constexpr (few5(Q).cost > 0) {
                if (take_few(E, EB, few5(Q)))
                    return bk5_launch<Q, few5(Q).eb, 6, L, true, few5(Q).dpar, GS>(prm, E, u, G, mass, lambda, v, s);
            }
            return bk5_launch<Q, EB, 6, L, true, DP, GS>(prm, E, u, G, mass, lambda, v, s);
        };
        if (gform == BK_G_FF) {
            if constexpr (eng_is_ff()) return go(ff2{});
            return BK_ERR_PREC;
        }
        return go(typename Eng::S{});
    }
    if (gform != BK_G_STORAGE) return BK_ERR_PREC;   // split G: even-odd D (GLL points), 6 factors
    if (F == 6) return bk5_launch<Q, fit_eb5<Q, 6, sweep_eb5(Q)>(), 6, L, false, 0>(prm, E, u, G, mass, lambda, v, s);
    if (F == 9) return bk5_launch<Q, fit_eb5<Q, 9, sweep_eb5(Q)>(), 9, L, false, 0>(prm, E, u, G, mass, lambda, v, s);
    return BK_ERR_PREC;
}
#endif  // BK_OP_TU == 5

#if BK_OP_TU == 6
// Column kernel: stage buffers.  With G read straight from HBM (FP32 storage,
// column layout) only u is staged, and one buffer leaves room for more blocks
// (q = 6 with the mass term 230 -> 224 us, q = 4 180 -> 177); the FP32-storage
// forms of the other layouts, and of nine factors, take two, the FP64 engines,
// ALU-bound, one.
constexpr bool col_gdir() { return sizeof(typename Eng::S) == 4 && BK_LAYOUT_TU == 2; }
constexpr int col_nbuf(int f) { return sizeof(typename Eng::S) == 4 && !(col_gdir() && f == 6) ? 2 : 1; }
// Elements per block: about 128 columns.
constexpr int col_eb_128(int q) { return (q * q >= 64) ? ((sizeof(typename Eng::S) == 4) ? 2 : 1) : (128 + q * q - 1) / (q * q); }
// The default: with six factors straight from HBM the fastest measured at about
// 2^25 points with the mass term (us, about 128 columns -> this): q = 3 265 ->
// 252, q = 4 188 -> 177, q = 5 250 -> 241, q = 6 240 -> 224, q = 7 281 -> 265,
// q = 8 234 -> 210, q = 9 362 -> 318.  Not with nine factors, whose loads bound
// the blocks otherwise.
constexpr int col_eb(int q, int f)
{
    constexpr int t[8] = {32, 7, 4, 5, 3, 1, 1, 1};   // q = 2..9
    return col_gdir() && f == 6 ? t[q - 2] : col_eb_128(q);
}

template <int Q, int EB, int F, int LAYOUT, int NBUF>
int bk5col_q(const double* D, long long E, const void* u, const void* G, const void* mass, double lambda, void* v,
             cudaStream_t s)
{
    using Cfg = BK5ColCfg<Eng, Q, EB, F, NBUF, LAYOUT>;
    using S = typename Eng::S;
    static_assert(Cfg::SMEM <= 232448, "BK5 block exceeds the shared memory of an SM");
    P5<typename Eng::C, Q> prm;
    for (int i = 0; i < Q * Q; ++i) prm.D[i] = Eng::coef(D[i]);
    auto kern = bk5_col_kernel<Eng, Q, EB, F, LAYOUT, NBUF>;
    const int occ = prepare<Cfg>(kern, Cfg::SMEM, Cfg::NT);
    if (occ <= 0) return BK_ERR_CUDA;
    const int grid = grid_for((E + EB - 1) / EB, occ);
    kern<<<grid, Cfg::NT, Cfg::SMEM, s>>>(prm, E, static_cast<const S*>(u), static_cast<const S*>(G),
                                          static_cast<const S*>(mass), lambda, static_cast<S*>(v), dev_ctx());
    return cudaGetLastError() == cudaSuccess ? BK_OK : BK_ERR_CUDA;
}

template <int Q>
int bk5col_f(int F, int eb, const double* D, long long E, const void* u, const void* G, const void* mass,
             double lambda, void* v, cudaStream_t s)
{
    // the option names the default or about 128 columns, and gets what it names
    constexpr int NB = col_nbuf(6);
    constexpr int EB0 = col_eb(Q, 6);
    constexpr int EB1 = col_eb_128(Q);
    static_assert(col_eb(Q, 9) == EB1, "nine factors have one number");
    if (F != 6 && F != 9) return BK_ERR_PREC;
    if (eb == 0) eb = F == 6 ? EB0 : EB1;
    if (eb != EB1 && (F == 9 || eb != EB0)) return BK_ERR_ARG;
    if (F == 9) return bk5col_q<Q, EB1, 9, BK_LAYOUT_TU, col_nbuf(9)>(D, E, u, G, mass, lambda, v, s);
    if (eb == EB0) return bk5col_q<Q, EB0, 6, BK_LAYOUT_TU, NB>(D, E, u, G, mass, lambda, v, s);
    return bk5col_q<Q, EB1, 6, BK_LAYOUT_TU, NB>(D, E, u, G, mass, lambda, v, s);
}
#endif  // BK_OP_TU == 6

#if BK_OP_TU == 1
template <int Q>
int bk1_q(const double* B, long long E, const void* jxw, const void* u, void* v, int jxw_t, cudaStream_t s)
{
    using S = typename Eng::S;
    P13<typename Eng::C, Q> prm;
    for (int i = 0; i < (Q - 1) * Q; ++i) prm.B[i] = Eng::coef(B[i]);
    for (int i = 0; i < Q * Q; ++i) prm.D[i] = Eng::coef(0.0);
    // the even-odd interpolation when B is centro-symmetric (GLL nodes,
    // Gauss points)
    const bool eo = make_eor<typename Eng::C, Q, Q - 1>(B, Q, true, +1, prm.bi, &Eng::coef) &&
                    make_eor<typename Eng::C, Q - 1, Q>(B, Q, false, +1, prm.bb, &Eng::coef);
    auto go = [&](auto e, auto n) {
        constexpr bool EO = decltype(e)::value;
        constexpr int EB = decltype(n)::value;
        using Cfg = BK1Cfg<Eng, Q, EB>;
        static_assert(Cfg::SMEM <= 232448, "BK1 block exceeds the shared memory of an SM");
        return launch_walk<Cfg, EO, EB>(&bk1_kernel<Eng, Q, EB, EO, false>, &bk1_kernel<Eng, Q, EB, EO, EO>, E, s, prm, E,
                                        static_cast<const S*>(u), static_cast<const S*>(jxw), jxw_t,
                                        static_cast<S*>(v));
    };
    using Large = std::integral_constant<int, sweep_eb1(Q)>;
    if (!eo) return go(std::false_type{}, std::integral_constant<int, gen_eb1(Q)>{});
    if constexpr (few1(Q).cost > 0) {
        if (take_few(E, Large::value, few1(Q)))
            return go(std::true_type{}, std::integral_constant<int, few1(Q).eb>{});
    }
    return go(std::true_type{}, Large{});
}

#endif  // BK_OP_TU == 1

#if BK_OP_TU == 3
template <int Q, int EB, bool EO, int DPAR, class GS = typename Eng::S>
int bk3_launch(const P13<typename Eng::C, Q>& prm, long long E, const void* G, const void* k, const void* u, void* v,
               cudaStream_t s)
{
    using Cfg = BK3Cfg<Eng, Q, EB, DPAR>;
    using S = typename Eng::S;
    static_assert(Cfg::SMEM <= 232448, "BK3 block exceeds the shared memory of an SM");
    // dynamic for the even-odd kernels, but not the float-float blocks of q = 9,
    // one to an SM, which nothing unbalances (765 us dealt against 787)
    constexpr bool DYN = EO && !(Q == 9 && DPAR != 0);
    return launch_walk<Cfg, EO, EB>(&bk3_kernel<Eng, Q, EB, EO, DPAR, GS, false>,
                                    &bk3_kernel<Eng, Q, EB, EO, DPAR, GS, DYN>, E, s, prm, E,
                                    static_cast<const S*>(u), static_cast<const GS*>(G), static_cast<const S*>(k),
                                    static_cast<S*>(v));
}

// direction-parallel gradient stages for the float-float engine from q = 7,
// with their own elements per block (us against one thread per line: q = 8
// 629 / 673, q = 10 763 / 1424, where a block is one element; q = 7 is level,
// 689 / 683, and keeps the shorter latency; q = 6 loses, 614 / 592)
constexpr bool sweep_dpar3(int q) { return eng_is_ff() && q >= 7; }
constexpr int sweep_eb3_dpar(int q) { return q == 9 ? 3 : 1; }

template <int Q, int EB>
int bk3_q(const double* B, const double* D, long long E, const void* G, const void* k, const void* u, void* v,
          int gform, cudaStream_t s)
{
    P13<typename Eng::C, Q> prm;
    for (int i = 0; i < (Q - 1) * Q; ++i) prm.B[i] = Eng::coef(B[i]);
    for (int i = 0; i < Q * Q; ++i) prm.D[i] = Eng::coef(D[i]);
    // the even-odd contractions when B is centro-symmetric and D
    // centro-antisymmetric (GLL nodes, Gauss points)
    const bool eo = make_p13_eo<typename Eng::C, Q>(prm, B, D, &Eng::coef);
    if (eo) {
        constexpr int DP = sweep_dpar3(Q) ? 2 : 0;
        constexpr int EBL = DP ? sweep_eb3_dpar(Q) : EB;
        // gs: G as stored, or split ahead of time (the float-float engine)
        auto go = [&](auto gs) {
            using GS = decltype(gs);
            if constexpr (few3(Q).cost > 0) {
                if (take_few(E, EBL, few3(Q)))
                    return bk3_launch<Q, few3(Q).eb, true, few3(Q).dpar, GS>(prm, E, G, k, u, v, s);
            }
            return bk3_launch<Q, EBL, true, DP, GS>(prm, E, G, k, u, v, s);
        };
        if (gform == BK_G_FF) {
            if constexpr (eng_is_ff()) return go(ff2{});
            return BK_ERR_PREC;
        }
        return go(typename Eng::S{});
    }
    if (gform != BK_G_STORAGE) return BK_ERR_PREC;   // split G: even-odd B and D (GLL nodes, Gauss points)
    return bk3_launch<Q, gen_eb3(Q), false, 0>(prm, E, G, k, u, v, s);
}

#endif  // BK_OP_TU == 3

#if BK_OP_TU == 7
template <int Q, int EB, bool EO, int DPAR, class GS = typename Eng::S>
int bk3adj_launch(const P13<typename Eng::C, Q>& prm, long long E, const void* G, const void* k, const void* u,
                  const void* res, void* dk, void* dG, cudaStream_t s)
{
    using Cfg = BK3AdjCfg<Eng, Q, EB, DPAR>;
    using S = typename Eng::S;
    static_assert(Cfg::SMEM <= 232448, "BK3 adjoint block exceeds the shared memory of an SM");
    return launch_walk<Cfg, EO, EB>(&bk3_adjoint_kernel<Eng, Q, EB, EO, DPAR, GS, false>,
                                    &bk3_adjoint_kernel<Eng, Q, EB, EO, DPAR, GS, EO>, E, s, prm, E,
                                    static_cast<const S*>(u), static_cast<const S*>(res), static_cast<const GS*>(G),
                                    static_cast<const S*>(k), static_cast<S*>(dk), static_cast<S*>(dG));
}

// the direction-parallel gradient sweeps for the float-float engine (q = 6
// 772 us against 930 with one thread per line, q = 10 1050 against 2845)
constexpr bool adj_dpar(int q) { return eng_is_ff() && q >= 6; }

template <int Q>
int bk3adj_q(const double* B, const double* D, long long E, const void* G, const void* k, const void* u,
             const void* res, void* dk, void* dG, int gform, cudaStream_t s)
{
    constexpr int EB = adj_eb(Q);
    P13<typename Eng::C, Q> prm;
    for (int i = 0; i < (Q - 1) * Q; ++i) prm.B[i] = Eng::coef(B[i]);
    for (int i = 0; i < Q * Q; ++i) prm.D[i] = Eng::coef(D[i]);
    if (make_p13_eo<typename Eng::C, Q>(prm, B, D, &Eng::coef)) {
        constexpr int DP = adj_dpar(Q) ? 2 : 0;
        // gs: G as stored, or split ahead of time (the float-float engine)
        auto go = [&](auto gs) {
            using GS = decltype(gs);
            if constexpr (few_adj(Q).cost > 0) {
                if (take_few(E, EB, few_adj(Q)))
                    return bk3adj_launch<Q, few_adj(Q).eb, true, few_adj(Q).dpar, GS>(prm, E, G, k, u, res, dk, dG, s);
            }
            return bk3adj_launch<Q, EB, true, DP, GS>(prm, E, G, k, u, res, dk, dG, s);
        };
        if (gform == BK_G_FF) {
            if constexpr (eng_is_ff()) return go(ff2{});
            return BK_ERR_PREC;
        }
        return go(typename Eng::S{});
    }
    if (gform != BK_G_STORAGE) return BK_ERR_PREC;
    return bk3adj_launch<Q, EB, false, 0>(prm, E, G, k, u, res, dk, dG, s);
}
#endif  // BK_OP_TU == 7

}  // namespace BK_TU_NS
using namespace BK_TU_NS;

#if BK_OP_TU == 5
#define BK_CATS_(a, b, c) a##_##b##_L##c
#define BK_CATS(a, b, c) BK_CATS_(a, b, c)
int BK_CATS(bk5_sweep, BK_SFX, BK_LAYOUT_TU)(int p, int F, const double* D, long long E, const void* u,
                                              const void* G, const void* mass, double lambda, void* v, int gform,
                                              cudaStream_t s)
{
    switch (p + 1) {
        case 2: return bk5_sweep_q<2>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 3: return bk5_sweep_q<3>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 4: return bk5_sweep_q<4>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 5: return bk5_sweep_q<5>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 6: return bk5_sweep_q<6>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 7: return bk5_sweep_q<7>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 8: return bk5_sweep_q<8>(F, D, E, u, G, mass, lambda, v, gform, s);
        case 9: return bk5_sweep_q<9>(F, D, E, u, G, mass, lambda, v, gform, s);
        default: return BK_ERR_ORDER;
    }
}
#endif

#if BK_OP_TU == 6
#define BK_CAT3_(a, b, c) a##_##b##_L##c
#define BK_CAT3(a, b, c) BK_CAT3_(a, b, c)
int BK_CAT3(bk5_col, BK_SFX, BK_LAYOUT_TU)(int p, int F, int eb, const double* D, long long E, const void* u,
                                            const void* G, const void* mass, double lambda, void* v, cudaStream_t s)
{
    switch (p + 1) {
        case 2: return bk5col_f<2>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 3: return bk5col_f<3>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 4: return bk5col_f<4>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 5: return bk5col_f<5>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 6: return bk5col_f<6>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 7: return bk5col_f<7>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 8: return bk5col_f<8>(F, eb, D, E, u, G, mass, lambda, v, s);
        case 9: return bk5col_f<9>(F, eb, D, E, u, G, mass, lambda, v, s);
        default: return BK_ERR_ORDER;
    }
}
#endif

#if BK_OP_TU == 1
int BK_CAT(launch_bk1, BK_SFX)(int p, long long E, const double* B, const void* jxw, const void* u, void* v,
                                int eb, int jxw_t, cudaStream_t s)
{
    (void)eb;
    switch (p + 2) {
        case 3: return bk1_q<3>(B, E, jxw, u, v, jxw_t, s);
        case 4: return bk1_q<4>(B, E, jxw, u, v, jxw_t, s);
        case 5: return bk1_q<5>(B, E, jxw, u, v, jxw_t, s);
        case 6: return bk1_q<6>(B, E, jxw, u, v, jxw_t, s);
        case 7: return bk1_q<7>(B, E, jxw, u, v, jxw_t, s);
        case 8: return bk1_q<8>(B, E, jxw, u, v, jxw_t, s);
        case 9: return bk1_q<9>(B, E, jxw, u, v, jxw_t, s);
        case 10: return bk1_q<10>(B, E, jxw, u, v, jxw_t, s);
        default: return BK_ERR_ORDER;
    }
}

#endif

#if BK_OP_TU == 3
int BK_CAT(launch_bk3, BK_SFX)(int p, long long E, const double* B, const double* D, const void* G, const void* k,
                                const void* u, void* v, int eb, int gform, cudaStream_t s)
{
    (void)eb;
    switch (p + 2) {
        case 3: return bk3_q<3, sweep_eb3(3)>(B, D, E, G, k, u, v, gform, s);
        case 4: return bk3_q<4, sweep_eb3(4)>(B, D, E, G, k, u, v, gform, s);
        case 5: return bk3_q<5, sweep_eb3(5)>(B, D, E, G, k, u, v, gform, s);
        case 6: return bk3_q<6, sweep_eb3(6)>(B, D, E, G, k, u, v, gform, s);
        case 7: return bk3_q<7, sweep_eb3(7)>(B, D, E, G, k, u, v, gform, s);
        case 8: return bk3_q<8, sweep_eb3(8)>(B, D, E, G, k, u, v, gform, s);
        case 9: return bk3_q<9, sweep_eb3(9)>(B, D, E, G, k, u, v, gform, s);
        case 10: return bk3_q<10, sweep_eb3(10)>(B, D, E, G, k, u, v, gform, s);
        default: return BK_ERR_ORDER;
    }
}

#endif

#if BK_OP_TU == 7
#define BK_CATL_(a, b, c) a##_##b##_L##c
#define BK_CATL(a, b, c) BK_CATL_(a, b, c)
// BK5 dispatch: kernel shape and G layout
int BK_CAT(launch_bk5, BK_SFX)(int p, long long E, const double* D, const void* G, const void* u, const void* mass,
                                double lambda, void* v, int F, int layout, int eb, int kernel, int gform,
                                cudaStream_t s)
{
    if (p < 1 || p > 8) return BK_ERR_ORDER;
    if (gform != BK_G_STORAGE && kernel == BK_KERNEL_COLUMN) return BK_ERR_PREC;   // sweep kernel only
    if (kernel == BK_KERNEL_SWEEP) {   // (AUTO is resolved by the caller, bk5_builtin_auto)
        switch (layout) {
            case 0: return BK_CATL(bk5_sweep, BK_SFX, 0)(p, F, D, E, u, G, mass, lambda, v, gform, s);
            case 1: return BK_CATL(bk5_sweep, BK_SFX, 1)(p, F, D, E, u, G, mass, lambda, v, gform, s);
            case 2: return BK_CATL(bk5_sweep, BK_SFX, 2)(p, F, D, E, u, G, mass, lambda, v, gform, s);
            default: return BK_ERR_PREC;
        }
    }
    switch (layout) {
        case 0: return BK_CATL(bk5_col, BK_SFX, 0)(p, F, eb, D, E, u, G, mass, lambda, v, s);
        case 1: return BK_CATL(bk5_col, BK_SFX, 1)(p, F, eb, D, E, u, G, mass, lambda, v, s);
        case 2: return BK_CATL(bk5_col, BK_SFX, 2)(p, F, eb, D, E, u, G, mass, lambda, v, s);
        default: return BK_ERR_PREC;
    }
}

int BK_CAT(launch_bk3_adjoint, BK_SFX)(int p, long long E, const double* B, const double* D, const void* G,
                                        const void* k, const void* u, const void* res, void* dk, void* dG,
                                        int gform, cudaStream_t s)
{
    switch (p + 2) {
        case 3: return bk3adj_q<3>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 4: return bk3adj_q<4>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 5: return bk3adj_q<5>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 6: return bk3adj_q<6>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 7: return bk3adj_q<7>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 8: return bk3adj_q<8>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 9: return bk3adj_q<9>(B, D, E, G, k, u, res, dk, dG, gform, s);
        case 10: return bk3adj_q<10>(B, D, E, G, k, u, res, dk, dG, gform, s);
        default: return BK_ERR_ORDER;
    }
}
#endif

}  // namespace bkg
