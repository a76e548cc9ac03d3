// FP64 metric epilogue on the device: the printed value of every cell of a lower
// triangle of counters (a matrix of `kssd3a ani --format matrix|triangle`), in the
// reference's formulas and operation order (lm3ways distance src/model_ani.h:285-305,
// naive and p distances src/command_ani.h:202-232, Mash/AAF
// src/command_ani.c:164-188, the 160-tree calibration src/model_refaf_hgb.h:7593-7628,
// metric selection src/command_ani.c:1129-1379, matrix exception values :1448-1456).
//
// This file is compiled with --fmad=false: no multiply-add is contracted, and every
// + - * / is the IEEE double operation the reference's host code performs, so every
// value built from them alone is bit-identical.  Only log, log1p and pow (CUDA's, not
// the host libm's) can differ in the last bits.  A cell's printed value is therefore the
// reference's unless it depends on one of them and either
//   - a calibration feature derived from them lies within kTol of a tree threshold on
//     the cell's path (a different leaf is then possible), or
//   - the value itself is derived from them (Naive, Mash or AAF metrics) and lies
//     within kTolValue of a rounding boundary of the six printed decimals (or of zero);
// such cells are listed for the host, which recomputes them with its own libm.
#include <cuda_pipeline.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "kssd_metric.cuh"

#ifndef KSSD_NUM_CODENS
#define KSSD_NUM_CODENS 11
#endif

namespace kssd {
namespace {

constexpr double kEps = 1e-8;
constexpr double kNaiveTau = 0.01;
// far above the few-ulp differences of two libms' log / log1p / pow on these values:
// relative distance of a calibration feature to a tree threshold, and distance (relative
// above 1) of a value to a rounding boundary of its printed decimals
constexpr double kTol = 1e-9;
constexpr double kTolValue = 1e-12;

// Trained constants of the reference's builds (src/model_ani.h:9-205): the 11-coden
// set, or the set its 9- and 10-coden builds share.
#if KSSD_NUM_CODENS < 11
__constant__ double c_denom[12] = {1.0090536851341, 1.0013604061893, 1.03540226374509, 1.04270754727088,
                                   1.0108940845453, 1.0010797461052, 0.98914550652945, 1.01536320288592,
                                   1.0061957741437, 0.9957814716168, 0.98352379677340, 1.00951820561544};
__constant__ double c_denom95[12] = {1.0196821174688, 0.9817771341602, 1.04637038371202, 1.02441485561367,
                                     1.0163855061091, 0.9824051281495, 1.04908985213703, 1.01102197270052,
                                     1.0074050784795, 1.0018402553389, 0.94654127396428, 0.94051319172603};
__constant__ double c_coef[17] = {-0.587100397752123, -7.93027271403258e-08, 4.98481429879899e-06,
                                  -1.63903694463017e-05, -4.93356600478016e-06, -14843.5350131617,
                                  306478.144745683,  -290254.345158429, -1781.00695309133,
                                  -1091.99589131905, 327.6575530681,    47395.255680747,
                                  47798.7112013701,  -35574.6303634354, -45398.423188085,
                                  -46461.4920783106, 35045.3583333325};
__constant__ double c_coef95[17] = {10.7394186800999,  -2.92835943410177e-08, 1.66112325940088e-05,
                                    -3.48757817098253e-05, -1.82725607919882e-05, 3151.11534599359,
                                    -1300.37794535582, -1824.96575177919, -21820.9227396359,
                                    -30943.09511694,   10100.3465983902,  25441.8492675468,
                                    35763.8363380932,  -3901.01958522226, -3669.6748819999,
                                    -4909.59256464219, -5653.59698386914};
constexpr double kNaiveScale = 0.1557143;
constexpr double kNaiveIntercept = 9.961e-5;
#else
__constant__ double c_denom[12] = {1.0178887, 1.0135146, 1.0302181, 1.1205122, 1.0136223, 0.9803396,
                                   1.0021964, 0.9839395, 0.9988935, 0.9690589, 0.9888171, 0.9817371};
__constant__ double c_denom95[12] = {1.0145656, 1.2708196, 1.2169829, 0.3904416, 0.8147527, 1.3389150,
                                     2.0581364, -1.4624736, 1.6877678, 2.4390067, 0.7878482, 0.6697437};
__constant__ double c_coef[17] = {6.86905236142636,  -5.85271800517096e-08, 7.43351941016881e-06,
                                  -1.95859228059721e-05, -8.44336369105416e-06, -11726.5478433625,
                                  -111109.682632437, 121000.895632267,  -741.538955661909,
                                  -1894.53741972785, 2585.81964981999,  -7744.5216892858,
                                  -18190.2514369096, 23306.3090989115,  8352.82760552325,
                                  19782.4294837312,  -25518.2493259614};
__constant__ double c_coef95[17] = {-1.69173585242774, -3.64716315423252e-08, 2.85880264052975e-05,
                                    -5.5597924264054e-05, -2.96208613804271e-05, 1106.96550282022,
                                    -83.197177767225,  -1671.88720051458, 152.75590068948,
                                    212.734805232395,  208.388739816682,  -0.27860125939004,
                                    2.27065806912198,  -10.2977013026837, -250.681324281127,
                                    -403.751360812353, -137.96628693833};
constexpr double kNaiveScale = 0.1544286;
constexpr double kNaiveIntercept = 7.133e-4;
#endif
struct Feat {
    uint32_t xny, section, mut2, diff;
};

__device__ double fold_scale(int drfold)
{
    const int delta = drfold - 8;
    if (delta < -60)
        return ldexp(1.0, -60);
    if (delta > 60)
        return ldexp(1.0, 60);
    return ldexp(1.0, delta);
}

__device__ double lm3_core(double X, double S, double M, double D, const double *p, const double *c)
{
    const double d1 = 1 / (p[0] * X + p[1] * S + p[2] * M + p[3] * D + kEps);
    const double d2 = 1 / (p[4] * X + p[5] * S + p[6] * M + p[7] * D + kEps);
    const double d3 = 1 / (p[8] * X + p[9] * S + p[10] * M + p[11] * D + kEps);
    return c[0] + c[1] * X + c[2] * S + c[3] * M + c[4] * D + c[5] * d1 + c[6] * d2 + c[7] * d3 + c[8] * X * d1 +
           c[9] * S * d1 + c[10] * M * d1 + c[11] * X * d2 + c[12] * S * d2 + c[13] * M * d2 + c[14] * X * d3 +
           c[15] * S * d3 + c[16] * M * d3;
}

// lm3ways_dist_from_features (src/model_ani.h:285-305)
__device__ double lm3ways_dist(const Feat &f, int drfold)
{
    const double scale = fold_scale(drfold);
    const double X = (double)f.xny * scale;
    const double S = (double)f.section * scale;
    const double M = (double)f.mut2 * scale;
    const double D = (double)f.diff * scale;
    if (X <= 0.0)
        return 1;
    else if (D <= 0.0)
        return 0;
    double dist = lm3_core(X, S, M, D, c_denom, c_coef);
    if (dist < 0.05)
        dist = lm3_core(X, S, M, D, c_denom95, c_coef95);
    if (dist < 0)
        dist = 0;
    return dist;
}

// get_naive_dist (src/command_ani.h:202-224): pow, so not exact
__device__ double naive_dist(const Feat &f)
{
    if (f.xny == 0)
        return 1;
    const double ratio = (double)(f.section + kEps) / (f.diff + kEps);
    const double dist0 = (double)f.diff / (f.xny + f.diff);
    const double final_dist = 1 - pow((1 - dist0), ratio);
    if (final_dist <= 0)
        return 0;
    double w = final_dist / kNaiveTau;
    if (w > 1.0)
        w = 1.0;
    return final_dist * kNaiveScale + kNaiveIntercept * w;
}

// get_p_dist (src/command_ani.h:226-232)
__device__ double p_dist(const Feat &f, int obj_bits)
{
    if (f.xny == 0 || obj_bits == 0)
        return 1;
    return (double)f.section / ((double)f.xny * ((double)obj_bits / 2.0));
}

// get_mashD / get_aafD (src/command_matrix.c:26-33): log, so not exact
__device__ double mash_d(uint32_t K, uint32_t X, uint32_t Y, uint32_t XnY)
{
    const double j = (double)XnY / (X + Y - XnY);
    return (-log(2 * j / (1 + j)) / (K));
}
__device__ double aaf_d(uint32_t K, uint32_t X, uint32_t Y, uint32_t XnY)
{
    return (-log((double)XnY / (X < Y ? X : Y)) / (K));
}

__device__ double clamp01(double x) { return x < 0.0 ? 0.0 : (x > 1.0 ? 1.0 : x); }

__device__ bool near(double v, double t) { return fabs(v - t) <= kTol * fmax(1.0, fabs(t)); }

// the 9- and 10-coden builds carry no calibration model (raw ANI)
constexpr bool kCalibrate = KSSD_NUM_CODENS >= 11;

// The calibration trees' features of a cell (refaf_hgb_predict_ani,
// src/model_refaf_hgb.h:7593-7628): x[0..10], and the mask of those derived from log /
// log1p or from an inexact raw ANI, whose thresholds are compared with a tolerance.
__device__ uint32_t hgb_features(const MetricParams &P, double raw_ani, bool raw_unc, double ref_af, const Feat &f,
                                 double *x, int stride)
{
    raw_ani = clamp01(raw_ani);
    if (ref_af < 1e-12)
        ref_af = 1e-12;
    if (ref_af > 1.0)
        ref_af = 1.0;
    const double xd = (double)f.xny;
    const double ref_aaf_ani = clamp01(1.0 + log(ref_af) / 11.0);
    x[0 * stride] = raw_ani;
    x[1 * stride] = ref_af;
    x[2 * stride] = log1p(xd * fold_scale(P.drfold));
    x[3 * stride] = (double)f.diff / xd;
    x[4 * stride] = (double)f.section / xd;
    x[5 * stride] = (double)f.mut2 / xd;
    x[6 * stride] = ref_aaf_ani;
    x[7 * stride] = raw_ani - ref_aaf_ani;
    x[8 * stride] = ref_af < 0.2 ? 1.0 : 0.0;
    x[9 * stride] = (ref_af >= 0.2 && ref_af < 0.5) ? 1.0 : 0.0;
    x[10 * stride] = ref_af >= 0.5 ? 1.0 : 0.0;
    return (1u << 2) | (1u << 6) | (1u << 7) | (raw_unc ? 1u : 0u);
}

// The trees' node records, from the CTA's copy in shared memory or from global memory.
template <bool SHARED>
__device__ __forceinline__ HgbNode load_node(const uint4 *nodes, uint32_t i)
{
    const uint4 w = SHARED ? nodes[i] : __ldg(nodes + i);
    HgbNode n;
    n.x = __longlong_as_double((long long)(((unsigned long long)w.y << 32) | w.x));
    n.feature = (signed char)(w.z & 0xFFu);
    n.flags = (unsigned char)((w.z >> 8) & 0xFFu);
    n.left = (unsigned short)(w.z >> 16);
    n.right = (unsigned short)(w.w & 0xFFFFu);
    return n;
}

// Walks kWays trees side by side, t0, t0 + step, ...: every round loads one node of each,
// and those loads are independent.  leaf[k] receives the leaf's node number (of a tree
// below P.ntrees), a number below P.nnodes in any case.  Returns true when a feature of `unc` came within kTol of a threshold
// on a path, or a walk did not end on a leaf (a malformed model): another leaf is
// possible, the cell is left to the host.
template <bool SHARED, int kWays>
__device__ __forceinline__ bool walk_trees(const MetricParams &P, const uint4 *nodes, int t0, int step,
                                           const double *x, int stride, uint32_t unc, uint32_t (&leaf)[kWays])
{
    uint32_t begin[kWays];
    uint32_t open = 0;
    bool bad = false;
#pragma unroll
    for (int k = 0; k < kWays; ++k) {
        const int t = t0 + k * step;
        begin[k] = t < P.ntrees ? __ldg(P.tree_begin + t) : 0u;
        leaf[k] = begin[k];
        open |= t < P.ntrees ? 1u << k : 0u;
    }
    for (int depth = 0; open && depth <= 64; ++depth) {  // trees are far shallower; the bound ends any walk
        HgbNode nd[kWays];
#pragma unroll
        for (int k = 0; k < kWays; ++k) {
            if (leaf[k] >= P.nnodes) {  // a malformed model
                bad = true;
                leaf[k] = 0;
                open &= ~(1u << k);
            }
            nd[k] = load_node<SHARED>(nodes, leaf[k]);
        }
#pragma unroll
        for (int k = 0; k < kWays; ++k) {
            if (nd[k].flags & 1u)
                open &= ~(1u << k);
            if ((open >> k) & 1u) {
                const double v = x[nd[k].feature * stride];
                if (((unc >> nd[k].feature) & 1u) && near(v, nd[k].x))
                    bad = true;
                const int left = isnan(v) ? (nd[k].flags >> 1) & 1u : (v <= nd[k].x);
                leaf[k] = begin[k] + (left ? nd[k].left : nd[k].right);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kWays; ++k)
        if ((open >> k) & 1u)  // the last step's node was not looked at: it may lie past the model
            leaf[k] = 0;
    return bad || open;
}

__device__ bool value_available(double v) { return v > 0.0 && v <= 1.0; }

// The calibrated ANI of a cell, once its trees have been walked.
struct Calibrated {
    double ani;
    bool path_unc;
};

// What a cell needs before its trees (raw ANI, AF of the reference side).
struct RawAni {
    double ani, af_r;
    bool unc;
};

// kssd_pair_metric for a matrix cell (ani_matrix_pair_value / ani_indexed_self_pair_metric,
// src/command_ani.c:1458-1496, 1627-1655, with make_selected_output_row :1349-1379), each
// intermediate evaluated only where the selected metric reads it.  A cell whose value
// depends on the calibration trees returns with *raw filled and *trees set when cal is
// null; the caller walks the trees and calls again with their sum.
__device__ __forceinline__ double pair_metric(const MetricParams &P, const Feat &f0, uint32_t qctx, uint32_t rctx,
                              const Calibrated *cal, RawAni *raw, bool *trees, bool *unc)
{
    if (qctx == 0 || rctx == 0)
        return P.s < 0 ? 1.0 - P.e : (double)P.e;
    const double af_q = (double)f0.xny / (double)qctx;
    const double af_r = (double)f0.xny / (double)rctx;
    const bool af_pass = (af_q > af_r ? af_q : af_r) >= (double)P.afcut;
    // effective metric (src/command_ani.c:1186-1347)
    int s = P.s < 0 ? -P.s : P.s;
    if (s < 1 || s > 9)
        s = 1;
    if (P.unassembled && !P.unified_metric && s <= 4)
        s = 4;
    const bool calibrates = s <= 2 && !P.raw_output && af_pass && !P.unassembled;
    double moe = P.e, naive = P.e;
    if (af_pass && !(P.v && calibrates) && (s <= 3 || s == 7 || s == 8))
        moe = lm3ways_dist(f0, P.drfold);
    const bool naive_unc = af_pass;
    if (af_pass && (s == 4 || (P.v && calibrates)))
        naive = naive_dist(f0);
    // fill_calibration (src/command_ani.c:1129-1184); matrix outputs never take the
    // assembly best-ANI guard (detail output only), so best ANI = calibrated ANI
    double calibrated = 0;
    bool cal_unc = false;
    if (calibrates) {
        const double ani = 1.0 - (P.v ? naive : moe);
        const bool ani_unc = P.v && naive_unc;
        if (f0.xny > 0 && f0.diff == 0 && f0.section == 0 && f0.mut2 == 0 && af_q == 1.0 && af_r == 1.0) {
            calibrated = 1.0;
        } else if (!kCalibrate || f0.xny == 0) {  // no calibration model, or nothing to calibrate: the raw ANI
            calibrated = ani;
            cal_unc = ani_unc;
        } else if (!cal) {
            *raw = RawAni{ani, af_r, ani_unc};
            *trees = true;
            return 0;
        } else {
            calibrated = cal->ani;
            if (cal->path_unc)
                *unc = true;  // another leaf is possible
        }
        if (cal_unc && (near(calibrated, 0.0) || near(calibrated, 1.0)))
            *unc = true;  // value_available() of an inexact calibrated value
    }
    if (s <= 2 && P.unassembled && P.v && af_pass && !P.raw_output) {
        // --qraw with the unified metric: the naive ANI stands in for the calibrated one, and
        // the selection below asks whether it lies in (0, 1]
        const double ani = 1.0 - naive_dist(f0);
        if (near(ani, 0.0) || near(ani, 1.0))
            *unc = true;
    }
    const bool available = calibrates && value_available(calibrated);
    if (s <= 2 && !available) {
        s = 3;
        if (P.v && af_pass && calibrates)  // moe was not needed until here
            moe = lm3ways_dist(f0, P.drfold);
    }
    const uint32_t K = (uint32_t)(P.ctx_bits / 2);
    double metric;
    bool vu = false;
    switch (s) {
    case 1:
    case 2: metric = 1.0 - calibrated; vu = cal_unc; break;
    case 3: metric = moe; break;
    case 4: metric = naive; vu = naive_unc; break;
    case 5: metric = mash_d(K, rctx, qctx, f0.xny); vu = true; break;
    case 6: metric = aaf_d(K, rctx, qctx, f0.xny); vu = true; break;
    case 7: metric = af_pass ? moe : mash_d(K, rctx, qctx, f0.xny); vu = !af_pass; break;
    case 8: metric = af_pass ? moe : aaf_d(K, rctx, qctx, f0.xny); vu = !af_pass; break;
    default: metric = af_pass ? p_dist(f0, P.obj_bits) : (double)P.e; break;
    }
    const double value = P.s < 0 ? 1.0 - metric : metric;
    if (vu) {
        // an inexact value prints the same six decimals unless it lies next to a rounding
        // boundary, or -- as 1 - distance, which may fall on either side of zero -- next to
        // zero, whose sign "%lf" prints (the distances themselves are never negative)
        const double y = fabs(value) * 1000000.0 + 0.5;
        if (!isfinite(value) || fabs(y - rint(y)) <= kTolValue * 1000000.0 * fmax(1.0, fabs(value)) ||
            (P.s < 0 && fabs(value) <= kTolValue))
            *unc = true;
    }
    return value;
}

// Row of triangle cell c: the largest q with q (q - 1) / 2 <= c (c < 2^39).
__device__ __forceinline__ uint32_t cell_row(size_t c)
{
    uint32_t q = (uint32_t)((1.0 + sqrt(1.0 + 8.0 * (double)c)) * 0.5);
    while ((size_t)q * (q - 1) / 2 > c)
        --q;
    while ((size_t)(q + 1) * q / 2 <= c)
        ++q;
    return q;
}

__device__ __forceinline__ Feat cell_feat(unsigned long long c, unsigned long long o)
{
    Feat f;
    f.xny = (uint32_t)c;
    f.mut2 = (uint32_t)(c >> 32);
    f.diff = (uint32_t)o;
    f.section = (uint32_t)(o >> 32);
    return f;
}

constexpr int kMetricThreads = 512;    // one CTA per SM
constexpr int kMetricWarps = kMetricThreads / 32;
constexpr uint32_t kMetricMost = 8;    // rounds of 32 cells in a warp's tile, at most; their loads are in flight together
constexpr int kWarpWays = 5;           // trees a lane walks side by side: 160 trees are one round of a warp
constexpr int kWarpCells = 12;         // from this many tree cells among 32 on, every lane walks its own
constexpr int kWarpSlots = 8;          // tree cells of a warp in flight
constexpr size_t kMetricSmem = 220 * 1024;

// Dynamic shared memory: the trees' nodes (SHARED), then each warp's area: per slot the
// features and the leaf numbers of one cell, or the features of 32 cells, one column a
// lane (a lane reads a feature that its node names: any choice of rows is free of bank
// conflicts, where an array of the thread would lie in local memory).
__host__ __device__ __forceinline__ size_t metric_slot_bytes(int ntrees)
{
    return kFeatures * 8 + ((size_t)ntrees * 2 + 7) / 8 * 8;
}
__host__ __device__ __forceinline__ size_t metric_warp_bytes(int ntrees)
{
    const size_t slots = kWarpSlots * metric_slot_bytes(ntrees), columns = kFeatures * 32 * 8;
    return slots > columns ? slots : columns;
}
__host__ __device__ __forceinline__ size_t metric_smem(int ntrees, uint32_t nnodes, bool shared)
{
    return (shared ? (size_t)nnodes * 16 : 0) + kMetricWarps * metric_warp_bytes(ntrees);
}

// The calibrated value of a cell whose trees sum to cal.
__device__ __noinline__ double calibrated_value(const MetricParams &P, const Feat &f, uint32_t qc, uint32_t rc,
                                                const Calibrated &cal, bool *unc)
{
    if (value_available(cal.ani)) {  // the selected metric is 1 - calibrated
        *unc = cal.path_unc;
        const double metric = 1.0 - cal.ani;
        return P.s < 0 ? 1.0 - metric : metric;
    }
    RawAni raw;
    bool trees = false;
    return pair_metric(P, f, qc, rc, &cal, &raw, &trees, unc);
}

// The value of every cell of a triangle.  Work unit: a warp takes a tile of consecutive
// cells, 32 of them at a time (256 a tile in a large triangle, fewer when that would leave
// warps without work, down to 32); warps do not wait for one another.
//
// A cell that needs no calibration tree is valued by its lane at once: most cells of a
// matrix of several species share no context, and that part is a stream of the counters.
// A cell's 160 trees are independent walks of dependent loads, and the cells of one
// species lie far apart in a row, so a lane that walks them alone leaves its warp idle
// for all of them.  Up to kWarpCells of 32 cells the warp takes them one after another,
// every lane walking five trees side by side, and each cell's lane then adds its leaf
// values in tree order (the sum's roundings are the reference's).  Above that (a matrix of
// one species) every lane walks its own cell's trees.  A walk's loads depend on one
// another, so the model (156 KB) is copied into shared memory first: read through L1, a
// triangle of a few thousand cells waits for L2 at most levels of every walk.
//
// Measured (B200, one call with its launch; before: a CTA per row, a thread per cell):
// 3,000 genomes of 300 species (4.5 M cells, 13,500 through the trees) 460 -> 57 us,
// 8,000 genomes of 800 species (32 M cells) 1,346 -> 304 us, 60 genomes of six species
// 335 -> 45 us (the latency of one warp's cells), 900 genomes of one species (404,550
// cells, all through the trees) 1,702 -> 1,530 us (issue and shared-memory conflicts).
template <bool SHARED>
__global__ void __launch_bounds__(kMetricThreads, 1) k_lower_metric(const __grid_constant__ MetricParams P, size_t cells, uint32_t rounds,
                                                     int warp_cells,
                                                     const unsigned long long *__restrict__ lc,
                                                     const unsigned long long *__restrict__ lo,
                                                     const uint32_t *__restrict__ qcnt,
                                                     const uint32_t *__restrict__ rcnt, double *__restrict__ out,
                                                     RecheckCell *__restrict__ recheck, unsigned long long cap,
                                                     unsigned long long *__restrict__ nrecheck)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint4 *nodes = reinterpret_cast<const uint4 *>(P.nodes);
    unsigned char *slots = smem;
    if (SHARED) {
        uint4 *copy = reinterpret_cast<uint4 *>(smem);
        for (uint32_t i = threadIdx.x; i < P.nnodes; i += kMetricThreads)
            __pipeline_memcpy_async(copy + i, nodes + i, 16);
        __pipeline_commit();
        __pipeline_wait_prior(0);
        nodes = copy;
        slots += (size_t)P.nnodes * 16;
        __syncthreads();
    }
    const size_t slot_bytes = metric_slot_bytes(P.ntrees);
    slots += warp * metric_warp_bytes(warp_cells ? P.ntrees : 0);
    auto put = [&](size_t cell, unsigned long long c, unsigned long long o, double v, bool unc) {
        if (unc) {
            out[cell] = __longlong_as_double(0x7FF8000000000000ll);
            const unsigned long long slot = atomicAdd(nrecheck, 1ull);
            if (slot < cap)
                recheck[slot] = RecheckCell{(unsigned long long)cell, c, o};
        } else {
            out[cell] = v;
        }
    };
    const size_t tile = (size_t)rounds * 32;
    // consecutive tiles on different SMs, so that a small triangle uses all of them
    for (size_t base = ((size_t)warp * gridDim.x + blockIdx.x) * tile; base < cells;
         base += (size_t)gridDim.x * kMetricWarps * tile) {
        const size_t end = min(base + tile, cells);
        // the tile's context words, and every cell that takes the constant (no shared
        // context between samples with sketches; its object word is not read)
        unsigned rest = 0;  // rounds with another cell
        {
            const size_t first = min(base + lane, cells - 1);
            uint32_t q = cell_row(first), r = (uint32_t)(first - (size_t)q * (q - 1) / 2);
            unsigned long long w[kMetricMost];
#pragma unroll
            for (uint32_t j = 0; j < kMetricMost; ++j) {
                const size_t cell = base + 32 * j + lane;
                w[j] = cell < end ? __ldcs(lc + cell) : 0;
            }
#pragma unroll
            for (uint32_t j = 0; j < kMetricMost; ++j) {
                const size_t cell = base + 32 * j + lane;
                if (cell < end) {
                    if (P.zero_const && (uint32_t)w[j] == 0 && __ldg(qcnt + q) && __ldg(rcnt + r))
                        __stcs(out + cell, P.zero_value);
                    else
                        rest |= 1u << j;
                }
                r += 32;
                while (r >= q) {  // past the row's end: row q holds q cells
                    r -= q;
                    ++q;
                }
            }
        }
        for (unsigned rounds_left = __reduce_or_sync(0xFFFFFFFFu, rest); rounds_left; rounds_left &= rounds_left - 1) {
            const int j = __ffs(rounds_left) - 1;
            const bool in = (rest >> j) & 1u;
            const size_t cell = base + 32 * j + lane;
            unsigned long long c = 0, o = 0;
            uint32_t qc = 0, rc = 0;
            bool trees = false;
            RawAni raw{};
            Feat f{};
            if (in) {
                c = __ldg(lc + cell);
                o = __ldg(lo + cell);
                const uint32_t q = cell_row(cell), r = (uint32_t)(cell - (size_t)q * (q - 1) / 2);
                qc = __ldg(qcnt + q);
                rc = __ldg(rcnt + r);
                f = cell_feat(c, o);
                bool unc = false;
                const double v = pair_metric(P, f, qc, rc, nullptr, &raw, &trees, &unc);
                if (!trees)
                    put(cell, c, o, v, unc);
            }
            unsigned todo = __ballot_sync(0xFFFFFFFFu, trees);
            if (__popc(todo) >= warp_cells) {
                if (trees) {
                    double *x = reinterpret_cast<double *>(slots) + lane;
                    const uint32_t fu = hgb_features(P, raw.ani, raw.unc, raw.af_r, f, x, 32);
                    Calibrated cal{P.baseline, false};
                    for (int t = 0; t < P.ntrees; t += kWarpWays) {
                        uint32_t leaf[kWarpWays];
                        cal.path_unc |= walk_trees<SHARED, kWarpWays>(P, nodes, t, 1, x, 32, fu, leaf);
#pragma unroll
                        for (int k = 0; k < kWarpWays; ++k)
                            if (t + k < P.ntrees)
                                cal.ani += load_node<SHARED>(nodes, leaf[k]).x;
                    }
                    cal.ani = clamp01(cal.ani);
                    bool unc = false;
                    const double v = calibrated_value(P, f, qc, rc, cal, &unc);
                    put(cell, c, o, v, unc);
                }
                todo = 0;
                __syncwarp();  // the columns are rewritten by the next cells
            }
            while (todo) {
                // the next kWarpSlots cells, the lane of rank i among them in slot i
                unsigned group = 0;
                for (int i = 0; i < kWarpSlots && todo; ++i) {
                    group |= todo & (0u - todo);
                    todo &= todo - 1;
                }
                const bool mine = (group >> lane) & 1u;
                const int rank = __popc(group & ((1u << lane) - 1u));
                uint32_t fu = 0;
                if (mine)
                    fu = hgb_features(P, raw.ani, raw.unc, raw.af_r, f,
                                      reinterpret_cast<double *>(slots + rank * slot_bytes), 1);
                __syncwarp();
                bool bad = false;
                unsigned left = group;
                for (int i = 0; left; ++i, left &= left - 1) {
                    const int src = __ffs(left) - 1;
                    const uint32_t cu = __shfl_sync(0xFFFFFFFFu, fu, src);
                    const double *x = reinterpret_cast<const double *>(slots + i * slot_bytes);
                    unsigned short *leaves = reinterpret_cast<unsigned short *>(slots + i * slot_bytes + kFeatures * 8);
                    bool b = false;
                    for (int t = (int)lane; t < P.ntrees; t += 32 * kWarpWays) {
                        uint32_t leaf[kWarpWays];
                        b |= walk_trees<SHARED, kWarpWays>(P, nodes, t, 32, x, 1, cu, leaf);
#pragma unroll
                        for (int k = 0; k < kWarpWays; ++k)
                            if (t + 32 * k < P.ntrees)
                                leaves[t + 32 * k] = (unsigned short)leaf[k];
                    }
                    const bool any = __any_sync(0xFFFFFFFFu, b) != 0;
                    if ((int)lane == src)
                        bad = any;
                }
                __syncwarp();
                if (mine) {
                    const unsigned short *leaves =
                        reinterpret_cast<const unsigned short *>(slots + rank * slot_bytes + kFeatures * 8);
                    Calibrated cal{P.baseline, bad};
#pragma unroll 8
                    for (int t = 0; t < P.ntrees; ++t)
                        cal.ani += load_node<SHARED>(nodes, leaves[t]).x;
                    cal.ani = clamp01(cal.ani);
                    bool unc = false;
                    const double v = calibrated_value(P, f, qc, rc, cal, &unc);
                    put(cell, c, o, v, unc);
                }
                __syncwarp();  // the slots are rewritten by the next cells
            }
        }
    }
}

}  // namespace

cudaError_t lower_metric_launch(const MetricParams &P, int n, const unsigned long long *lc,
                                const unsigned long long *lo, const uint32_t *qcnt, const uint32_t *rcnt, double *out,
                                RecheckCell *recheck, unsigned long long cap, unsigned long long *nrecheck, int sms,
                                cudaStream_t st)
{
    if (n < 2)
        return cudaSuccess;
    const size_t cells = (size_t)n * (n - 1) / 2;
    const size_t warps = (size_t)sms * kMetricWarps;
    const size_t even = cells / (warps * 32);
    const uint32_t rounds = (uint32_t)(even < 1 ? 1 : even < kMetricMost ? even : kMetricMost);
    const size_t tiles = (cells + (size_t)rounds * 32 - 1) / ((size_t)rounds * 32);
    const unsigned grid = (unsigned)(tiles < (size_t)sms ? tiles : (size_t)sms);
    // the trees matter where the selected metric may be calibrated; a model too large for
    // shared memory is read from global memory
    const int s = P.s < 0 ? -P.s : P.s;
    MetricParams Q = P;
    if (s >= 3 && s <= 9)
        Q.ntrees = 0;
    const bool shared = Q.ntrees > 0 && !P.raw_output && !P.unassembled && Q.nnodes <= 65536 &&
                        metric_smem(Q.ntrees, Q.nnodes, true) <= kMetricSmem;
    // a model whose leaf numbers do not fit the slots: every lane walks its own cells
    const bool slots = metric_smem(Q.ntrees, Q.nnodes, shared) <= kMetricSmem && Q.nnodes <= 65536;
    const size_t smem = metric_smem(slots ? Q.ntrees : 0, Q.nnodes, shared);
    auto kern = shared ? k_lower_metric<true> : k_lower_metric<false>;
    // the limit is the context's: the same for every call, so that no thread lowers it before
    // another one's launch
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMetricSmem);
    if (e != cudaSuccess)
        return e;
    kern<<<grid, kMetricThreads, smem, st>>>(Q, cells, rounds, slots ? kWarpCells : 0, lc, lo, qcnt, rcnt, out, recheck, cap, nrecheck);
    return cudaGetLastError();
}

}  // namespace kssd
