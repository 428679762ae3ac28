// life_simulation_b200/csrc/lenia_fft_wide.cuh -- the compile-time-plan
// spectral passes for every transform length with factors 2, 3 and 5 that the
// catalogue (fft_fast_common.cuh) does not hold: column lengths 64..4096, half
// row lengths 32..2048, compiled in eight translation units.
//
// The runtime-plan kernels of lenia_fft.cu, which these lengths ran on before,
// divide by a runtime number for every element of every pass, take more passes
// (720 = 16 * 5 * 3 * 3, 405 = 5 * 3 * 3 * 3 * 3) and stage nothing ahead. They
// stay for lengths outside these ranges (a few rows, a field of 8192 columns)
// and for columns of 3000, 3125 and 3200, whose four passes spill here (0.9 to
// 0.96 of the runtime plan's speed, or five passes). A substep of three
// kernels, R = 24, back to back, runtime plan -> these: 1280 x 720 92 -> 26 us,
// 810 x 486 64 -> 19, 640 x 360 43 -> 13, 2560 x 1440 317 -> 93, 3840 x 2160
// 665 -> 193, 1250 x 1250 109 -> 55, 100 x 75 25 -> 10; over every length of the
// ranges 2.6 times on average.
#pragma once
#include "fft_passes.cuh"

namespace lenia {
namespace {

// The radices of a length, in forward order for columns and inverse order for
// rows (the last one is the pass whose values stay in registers): the fewest
// and cheapest passes. A pass costs its exchange through shared memory (8)
// plus what a large codelet adds in registers; the last radix sets the thread
// count (length / radix: at most 256 a transform where possible) and the registers held
// across the kernels, and is best at 8; a smaller radix than it leaves its
// pass with more items than threads. Lengths up to 256 could take two passes
// of 15 or 16 each, but two such codelets hold 60 registers a thread and halve
// the threads.
struct WideRadices {
    int np = 0;
    int r[4] = {1, 1, 1, 1};
    int cost = 1 << 20;
};
constexpr int wide_pass_cost(int r) { return 8 + (r <= 8 ? 0 : r <= 10 ? 1 : r == 12 ? 2 : 3); }
constexpr int wide_last_cost(int n, int r, int smallest) {
    return (r >= 15 ? 8 : r == 12 ? 6 : r == 10 ? 2 : r == 9 ? 1 : r == 8 ? 0 : r == 6 ? 1 : r == 5 ? 2 : r == 4 ? 3 : 6) +
           (n / r > 400 ? 12 : n / r > 256 ? 4 : 0) + (smallest < r ? (r > 8 ? 6 : 3) : 0);
}
constexpr int wide_min(int a, int b) { return a < b ? a : b; }
constexpr WideRadices wide_radices(int n) {
    constexpr int R[11] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
    WideRadices best;
    for (int a : R) {
        if (n % a != 0) continue;
        for (int b : R) {
            if ((n / a) % b != 0) continue;
            const int rest = n / a / b, ab = wide_pass_cost(a) + wide_pass_cost(b), mab = wide_min(a, b);
            const int two = ab + wide_last_cost(n, b, mab);
            if (rest == 1 && two < best.cost) best = WideRadices{2, {a, b, 1, 1}, two};
            for (int c : R) {
                if (rest % c != 0) continue;
                const int abc = ab + wide_pass_cost(c), mabc = wide_min(mab, c);
                const int three = abc + wide_last_cost(n, c, mabc);
                if (rest == c && three < best.cost) best = WideRadices{3, {a, b, c, 1}, three};
                for (int d : R) {
                    const int four = abc + wide_pass_cost(d) + wide_last_cost(n, d, wide_min(mabc, d));
                    if (rest == c * d && four < best.cost) best = WideRadices{4, {a, b, c, d}, four};
                }
            }
        }
    }
    return best;
}
template <int N, int NP>
struct WidePlanOf;
template <int N>
struct WidePlanOf<N, 2> {
    static constexpr WideRadices w = wide_radices(N);
    using type = Plan<w.r[0], w.r[1]>;
};
template <int N>
struct WidePlanOf<N, 3> {
    static constexpr WideRadices w = wide_radices(N);
    using type = Plan<w.r[0], w.r[1], w.r[2]>;
};
template <int N>
struct WidePlanOf<N, 4> {
    static constexpr WideRadices w = wide_radices(N);
    using type = Plan<w.r[0], w.r[1], w.r[2], w.r[3]>;
};
template <int N>
using WidePlan = typename WidePlanOf<N, wide_radices(N).np>::type;

// Columns and rows per CTA: the larger of two shapes keeps a CTA within 640
// (512) threads, the smaller (half of it) is for fields that would leave SMs
// idle.
template <class PF>
constexpr int wide_cols() {
    return 4 * (PF::n / PF::last()) <= 640 ? 4 : 2;
}
// Last-pass items per thread: two where two columns would still want more.
template <class PF>
constexpr int wide_split() {
    return wide_cols<PF>() * (PF::n / PF::last()) > 640 ? 2 : 1;
}
template <class PI>
constexpr int wide_rows() {
    return 4 * (PI::n / PI::last()) <= 512 ? 4 : 2 * (PI::n / PI::last()) <= 512 ? 2 : 1;
}

}  // namespace

#define LENIA_WIDE_COLS_0(X) \
    X(72) X(120) X(192) X(300) X(432) X(625) X(800) X(1152) X(1458) X(1920) X(2400) X(3072) X(3888)
#define LENIA_WIDE_COLS_1(X) \
    X(75) X(125) X(200) X(320) X(450) X(640) X(810) X(1200) X(1500) X(1944) X(2430) X(3240) X(4000)
#define LENIA_WIDE_COLS_2(X) \
    X(80) X(135) X(225) X(324) X(480) X(648) X(864) X(1215) X(1536) X(2000) X(2500) X(3375) X(4050)
#define LENIA_WIDE_COLS_3(X) \
    X(81) X(144) X(240) X(360) X(486) X(675) X(900) X(1250) X(1600) X(2025) X(2560) X(3456)
#define LENIA_WIDE_COLS_4(X) \
    X(90) X(150) X(243) X(375) X(500) X(720) X(960) X(1280) X(1620) X(2160) X(2592) X(3600)
#define LENIA_WIDE_COLS_5(X) \
    X(96) X(160) X(250) X(384) X(540) X(729) X(972) X(1296) X(1728) X(2187) X(2700) X(3645)
#define LENIA_WIDE_COLS_6(X) \
    X(100) X(162) X(270) X(400) X(576) X(750) X(1000) X(1350) X(1800) X(2250) X(2880) X(3750)
#define LENIA_WIDE_COLS_7(X) \
    X(108) X(180) X(288) X(405) X(600) X(768) X(1125) X(1440) X(1875) X(2304) X(2916) X(3840)
#define LENIA_WIDE_ROWS_0(X) \
    X(32) X(72) X(120) X(200) X(300) X(432) X(625) X(800) X(1125) X(1440) X(1875)
#define LENIA_WIDE_ROWS_1(X) \
    X(36) X(75) X(125) X(216) X(320) X(450) X(640) X(810) X(1152) X(1458) X(1920)
#define LENIA_WIDE_ROWS_2(X) \
    X(40) X(80) X(135) X(225) X(324) X(480) X(648) X(864) X(1200) X(1500) X(1944)
#define LENIA_WIDE_ROWS_3(X) \
    X(45) X(81) X(144) X(240) X(360) X(486) X(675) X(900) X(1215) X(1536) X(2000)
#define LENIA_WIDE_ROWS_4(X) \
    X(48) X(90) X(150) X(243) X(375) X(500) X(720) X(972) X(1250) X(1600) X(2025)
#define LENIA_WIDE_ROWS_5(X) \
    X(50) X(96) X(160) X(250) X(384) X(540) X(729) X(1000) X(1280) X(1620)
#define LENIA_WIDE_ROWS_6(X) \
    X(54) X(100) X(162) X(270) X(400) X(576) X(750) X(1024) X(1296) X(1728)
#define LENIA_WIDE_ROWS_7(X) \
    X(60) X(108) X(180) X(288) X(405) X(600) X(768) X(1080) X(1350) X(1800)

// Part p's lengths: plans, and launches (cudaErrorNotSupported for a length
// or shape it does not hold). `shape` 0: the larger number of columns or rows
// per CTA, 1: half of it.
#define LENIA_WIDE_DECLARE(p)                                                                                \
    bool wide_col_plan_##p(int H, FastPlan& forward_plan);                                                   \
    bool wide_row_plan_##p(int M, FastPlan& inverse_plan);                                                   \
    cudaError_t wide_col_##p(int H, int shape, const SpectralWorld& w, const FastTables& t, cudaStream_t s); \
    cudaError_t wide_row_##p(int M, int H, int shape, const SpectralWorld& w, const float2* tw_r2c,          \
                             const FastTables& t, cudaStream_t s);
#define LENIA_WIDE_EACH(F) F(0) F(1) F(2) F(3) F(4) F(5) F(6) F(7)
LENIA_WIDE_EACH(LENIA_WIDE_DECLARE)
#undef LENIA_WIDE_DECLARE
// The row passes of the catalogue's half rows under a wide column length
// (lenia_fft_wide_mixed.cu): the catalogue's plans, the wide lengths' growth map.
cudaError_t wide_row_mixed(int M, int H, int shape, const SpectralWorld& w, const float2* tw_r2c, const FastTables& t,
                           cudaStream_t s);

}  // namespace lenia
