// alias.cu -- alias-table build and sampling on the device.
//
// Two builds:
//  * reference mode: the pairing of DevilRay's generateAliasTable
//    (src/DistributionSamplers.cpp:39-149) -- a sequential float total and two
//    max-heaps ordered by p_A -- run by one thread with heaps whose sift
//    operations follow the standard binary-heap algorithm of the C++ library
//    the reference uses (push: sift the new element up while its parent
//    compares lower; pop: move the last element to the top position's hole
//    path along the larger child, preferring the right child on ties, then sift
//    up). Bit-identical to the reference; O(n log n) on one thread.
//  * sweep mode (default): the sweeping construction of Huebschle-Schneider
//    and Sanders ("Parallel Weighted Random Sampling", ACM TOMS 2022) in exact
//    fixed point (64-bit weights, 128-bit prefix sums), so it is order
//    independent and bit-identical to its CPU restatement in the oracle.
//    Slot i holds item i; lights are aliased to the heavy item whose surplus
//    covers them (prefix sums + binary search), heavies to the next heavy.

#include "dr_internal.h"
#include "alias_kernels.cuh"
#include "launch.cuh"

#include <cooperative_groups.h>

#include <climits>
#include <mutex>

namespace dr {

namespace cg = cooperative_groups;

using i128 = __int128;

// ---- reference-compatible build ------------------------------------------------

struct HeapItem {
    float p;
    int32_t a;
};

__host__ __device__ __forceinline__ void heap_push(HeapItem *h, int32_t &len, HeapItem v)
{
    int32_t hole = len++;
    int32_t parent = (hole - 1) / 2;
    while (hole > 0 && h[parent].p < v.p) {
        h[hole] = h[parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    h[hole] = v;
}

// Removes the top element (the caller read it before).
__host__ __device__ __forceinline__ void heap_pop(HeapItem *h, int32_t &len)
{
    if (len > 1) {
        const int32_t n = len - 1;  // size of the heap without the moved-out top
        const HeapItem value = h[n];
        h[n] = h[0];
        int32_t hole = 0, child = 0;
        while (child < (n - 1) / 2) {
            child = 2 * (child + 1);
            if (h[child].p < h[child - 1].p) --child;
            h[hole] = h[child];
            hole = child;
        }
        if ((n & 1) == 0 && child == (n - 2) / 2) {
            child = 2 * (child + 1);
            h[hole] = h[child - 1];
            hole = child - 1;
        }
        int32_t parent = (hole - 1) / 2;
        while (hole > 0 && h[parent].p < value.p) {
            h[hole] = h[parent];
            hole = parent;
            parent = (hole - 1) / 2;
        }
        h[hole] = value;
    }
    --len;
}

__host__ __device__ __forceinline__ void ensure_pa_larger(dr_alias_entry &e)
{
    if (e.p_A < 0.5f) {
        e.p_A = 1 - e.p_A;
        const int32_t t = e.A;
        e.A = e.B;
        e.B = t;
        const float f = e.pdf_A;
        e.pdf_A = e.pdf_B;
        e.pdf_B = f;
    }
}

// One table, one thread: filter, sequential total, heap pairing, entries in
// processing order, then the pdf fill (src/DistributionSamplers.cpp:39-149).
__device__ void alias_ref_build_one(const float *__restrict__ w, uint32_t n, dr_alias_entry *__restrict__ out,
                                    HeapItem *under, HeapItem *over, float *filtered, bool fill_pdfs,
                                    float *total_out)
{
    float total = 0.f;
    for (uint32_t i = 0; i < n; ++i) {
        const float fi = (0.f < w[i]) ? w[i] : 0.f;  // std::max(0.f, w[i])
        filtered[i] = fi;
        total = total + fi;
    }
    if (total_out) *total_out = total;
    if (n == 0) return;
    if (total < 1e-5f) {
        const float u = 1.0f / (float)n;
        for (uint32_t i = 0; i < n; ++i) out[i] = dr_alias_entry{1.0f, u, 0.0f, (int32_t)i, -1};
        return;
    }
    int32_t nu = 0, no = 0;
    uint32_t ptr = 0;
    const float fn = (float)n;
    for (uint32_t i = 0; i < n; ++i) {
        const float p = filtered[i] / total;
        const HeapItem e{fn * p, (int32_t)i};
        if (e.p > 1) heap_push(over, no, e);
        else if (e.p < 1) heap_push(under, nu, e);
        else out[ptr++] = dr_alias_entry{e.p, 0.f, 0.f, e.a, -1};
    }
    while (nu > 0 && no > 0) {
        HeapItem u = under[0];
        HeapItem o = over[0];
        heap_pop(under, nu);
        heap_pop(over, no);
        dr_alias_entry ue{u.p, 0.f, 0.f, u.a, o.a};
        o.p = o.p + u.p - 1;
        ensure_pa_larger(ue);
        out[ptr++] = ue;
        if (o.p > 1) heap_push(over, no, o);
        else if (o.p < 1) heap_push(under, nu, o);
        else {
            dr_alias_entry oe{o.p, 0.f, 0.f, o.a, -1};
            ensure_pa_larger(oe);
            out[ptr++] = oe;
        }
    }
    while (nu > 0) {
        const HeapItem e = under[0];
        heap_pop(under, nu);
        out[ptr++] = dr_alias_entry{1.0f, 0.f, 0.f, e.a, -1};
    }
    while (no > 0) {
        const HeapItem e = over[0];
        heap_pop(over, no);
        out[ptr++] = dr_alias_entry{1.0f, 0.f, 0.f, e.a, -1};
    }
    if (fill_pdfs) {
        for (uint32_t i = 0; i < n; ++i) {
            dr_alias_entry &e = out[i];
            e.pdf_A = filtered[e.A] / total;
            e.pdf_B = (e.B >= 0 && (uint32_t)e.B < n) ? filtered[e.B] / total : 0.0f;
        }
    }
}

__global__ void k_alias_ref_pair(const float *__restrict__ w, uint32_t n, dr_alias_entry *__restrict__ out,
                                 HeapItem *under, HeapItem *over, float *filtered, float *total_out)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    alias_ref_build_one(w, n, out, under, over, filtered, false, total_out);
}

// pdf fill (src/DistributionSamplers.cpp:135-146) of the single-table build, parallel.
__global__ void k_alias_ref_pdfs(uint32_t n, dr_alias_entry *__restrict__ out, const float *__restrict__ filtered,
                                 const float *__restrict__ total_in)
{
    const float total = *total_in;
    if (total < 1e-5f) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        dr_alias_entry e = out[i];
        e.pdf_A = filtered[e.A] / total;
        e.pdf_B = (e.B >= 0 && (uint32_t)e.B < n) ? filtered[e.B] / total : 0.0f;
        out[i] = e;
    }
}

// Many independent tables, one thread each: table s covers entries
// [begin[s], begin[s] + count[s]) of w and out (object-local indices).
__global__ void k_alias_ref_segments(const float *__restrict__ w, const uint32_t *__restrict__ begin,
                                     const uint32_t *__restrict__ count, uint32_t nseg,
                                     dr_alias_entry *__restrict__ out, HeapItem *heaps, float *filtered)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const uint32_t b = begin[s], n = count[s];
    alias_ref_build_one(w + b, n, out + b, heaps + 2 * (size_t)b, heaps + 2 * (size_t)b + n, filtered + b, true,
                        nullptr);
}

// ---- sweep build -----------------------------------------------------------------------

__device__ __forceinline__ float clamp_weight(float w) { return (w > 0.0f && isfinite(w)) ? w : 0.0f; }

__device__ __forceinline__ int float_exponent(float w)
{
    int e;
    frexpf(w, &e);
    return e;
}

// Warp-level inclusive scan of a 128-bit value.
__device__ __forceinline__ i128 warp_scan_i128(i128 v)
{
    const int lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long lo = (unsigned long long)v;
        const long long hi = (long long)(v >> 64);
        const unsigned long long lo_o = __shfl_up_sync(0xffffffffu, lo, off);
        const long long hi_o = __shfl_up_sync(0xffffffffu, hi, off);
        const i128 o = ((i128)hi_o << 64) | (i128)lo_o;
        if (lane >= off) v += o;
    }
    return v;
}

__device__ __forceinline__ int warp_scan_int(int v)
{
    const int lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += o;
    }
    return v;
}

// Block-wide exclusive scan of (count, D, S) triples; returns the block total
// through `total`. blockDim.x == kSweepBlock.
struct Agg {
    int32_t lights;
    int32_t pad;
    i128 D;
    i128 S;
};

__device__ Agg block_exclusive_scan(Agg v, Agg &total)
{
    __shared__ int s_cnt[kSweepBlock / 32];
    __shared__ i128 s_D[kSweepBlock / 32];
    __shared__ i128 s_S[kSweepBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c_inc = warp_scan_int(v.lights);
    const i128 d_inc = warp_scan_i128(v.D);
    const i128 s_inc = warp_scan_i128(v.S);
    if (lane == 31) {
        s_cnt[warp] = c_inc;
        s_D[warp] = d_inc;
        s_S[warp] = s_inc;
    }
    __syncthreads();
    if (warp == 0) {
        constexpr int nw = kSweepBlock / 32;
        int c = lane < nw ? s_cnt[lane] : 0;
        i128 d = lane < nw ? s_D[lane] : (i128)0;
        i128 s = lane < nw ? s_S[lane] : (i128)0;
        c = warp_scan_int(c);
        d = warp_scan_i128(d);
        s = warp_scan_i128(s);
        if (lane < nw) {
            s_cnt[lane] = c;
            s_D[lane] = d;
            s_S[lane] = s;
        }
    }
    __syncthreads();
    Agg out;
    const int c_before = warp > 0 ? s_cnt[warp - 1] : 0;
    const i128 d_before = warp > 0 ? s_D[warp - 1] : (i128)0;
    const i128 s_before = warp > 0 ? s_S[warp - 1] : (i128)0;
    out.lights = c_before + c_inc - v.lights;
    out.D = d_before + d_inc - v.D;
    out.S = s_before + s_inc - v.S;
    out.pad = 0;
    total.lights = s_cnt[kSweepBlock / 32 - 1];
    total.D = s_D[kSweepBlock / 32 - 1];
    total.S = s_S[kSweepBlock / 32 - 1];
    total.pad = 0;
    __syncthreads();
    return out;
}

struct SweepScalars {
    int emax;
    int lg;
    int shift;
    int uniform;
    unsigned long long W;
    int32_t num_lights;
    int32_t num_heavies;
    i128 D_total;
    double Wd, inv_W, nd;  // (double)W, 1 / Wd, (double)n
};

// floor(w 2^shift) of a clamped weight w = m 2^(e - 24), m its
// 24-bit significand (a denormal one has fewer bits; the value is the same).
__device__ __forceinline__ long long fixed_weight_bits(float w, int shift)
{
    const uint32_t bits = __float_as_uint(w);
    const int be = (int)(bits >> 23);
    const long long m = be ? (long long)((bits & 0x7fffffu) | 0x800000u) : (long long)(bits & 0x7fffffu);
    const int s = (be ? be : 1) - 150 + shift;
    return s >= 0 ? m << s : s > -64 ? m >> -s : 0;
}

// The same as a double, by its bits: an FP32 significand always fits, and the
// conversion from an integer would run at the FP64 rate.
__device__ __forceinline__ double fixed_weight_double(float w, int shift)
{
    const uint32_t bits = __float_as_uint(w), be = bits >> 23;
    if (be == 0) return (double)fixed_weight_bits(w, shift);
    const int s = (int)be - 150 + shift;  // shift of the 24-bit significand
    if (s <= -24) return 0.0;
    const uint32_t frac = (bits & 0x7fffffu) & (s < 0 ? ~0u << -s : ~0u);
    return __hiloint2double((int)(((be - 127 + 1023 + (uint32_t)shift) << 20) | (frac >> 3)), (int)(frac << 29));
}

__device__ __forceinline__ long long fixed_weight(float w, const SweepScalars &sc)
{
    if (sc.emax == INT_MIN) return 0;
    return fixed_weight_bits(clamp_weight(w), sc.shift);
}

__global__ void k_sweep_init(SweepScalars *sc, uint32_t n)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        sc->emax = INT_MIN;
        int lg = 0;
        while ((1ll << lg) < (long long)n + 1) ++lg;
        sc->lg = lg;
        sc->W = 0;
        sc->uniform = 0;
    }
}

__global__ void k_sweep_exponent(const float *__restrict__ w, uint32_t n, SweepScalars *sc)
{
    int e = INT_MIN;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float x = clamp_weight(w[i]);
        if (x > 0.0f) e = max(e, float_exponent(x));
    }
    for (int off = 16; off > 0; off >>= 1) e = max(e, __shfl_down_sync(0xffffffffu, e, off));
    if ((threadIdx.x & 31) == 0 && e != INT_MIN) atomicMax(&sc->emax, e);
}

__global__ void k_sweep_sum(const float *__restrict__ w, uint32_t n, SweepScalars *sc)
{
    __shared__ SweepScalars s;
    if (threadIdx.x == 0) {
        s = *sc;
        s.shift = 61 - s.lg - s.emax;
    }
    __syncthreads();
    unsigned long long acc = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        acc += (unsigned long long)fixed_weight(w[i], s);
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(&sc->W, acc);
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->shift = s.shift;
}

// Per tile of kSweepBlock items: (light count, deficit sum, surplus sum).
__global__ void k_sweep_tile_aggregates(const float *__restrict__ w, uint32_t n, const SweepScalars *sc, Agg *tiles)
{
    const SweepScalars s = *sc;
    const uint32_t i = blockIdx.x * kSweepBlock + threadIdx.x;
    Agg v{0, 0, 0, 0};
    if (i < n) {
        const long long a = (long long)n * fixed_weight(w[i], s) - (long long)s.W;
        if (a < 0) {
            v.lights = 1;
            v.D = (i128)(-a);
        } else {
            v.S = (i128)a;
        }
    }
    Agg total;
    block_exclusive_scan(v, total);
    if (threadIdx.x == 0) tiles[blockIdx.x] = total;
}

// One block: exclusive scan over the tile aggregates (in place).
__global__ void k_sweep_scan_tiles(Agg *tiles, uint32_t num_tiles, SweepScalars *sc, uint32_t n)
{
    Agg carry{0, 0, 0, 0};
    for (uint32_t base = 0; base < num_tiles; base += kSweepBlock) {
        const uint32_t t = base + threadIdx.x;
        Agg v = t < num_tiles ? tiles[t] : Agg{0, 0, 0, 0};
        Agg total;
        Agg ex = block_exclusive_scan(v, total);
        if (t < num_tiles) {
            Agg o;
            o.lights = carry.lights + ex.lights;
            o.D = carry.D + ex.D;
            o.S = carry.S + ex.S;
            o.pad = 0;
            tiles[t] = o;
        }
        carry.lights += total.lights;
        carry.D += total.D;
        carry.S += total.S;
    }
    if (threadIdx.x == 0) {
        sc->num_lights = carry.lights;
        sc->num_heavies = (int32_t)n - carry.lights;
        sc->D_total = carry.D;
        sc->Wd = (double)sc->W;
        sc->inv_W = 1.0 / sc->Wd;
        sc->nd = (double)n;
        const float Wf = sc->emax == INT_MIN ? 0.0f : (float)ldexp((double)sc->W, -sc->shift);
        sc->uniform = !(Wf >= 1e-5f);
    }
}

// Writes the light / heavy lists in index order with their running sums.
__global__ void k_sweep_scatter(const float *__restrict__ w, uint32_t n, const SweepScalars *sc, const Agg *tiles,
                                int32_t *lights, i128 *Dexcl, int32_t *heavies, i128 *Sincl)
{
    const SweepScalars s = *sc;
    const uint32_t i = blockIdx.x * kSweepBlock + threadIdx.x;
    Agg v{0, 0, 0, 0};
    long long a = 0;
    if (i < n) {
        a = (long long)n * fixed_weight(w[i], s) - (long long)s.W;
        if (a < 0) {
            v.lights = 1;
            v.D = (i128)(-a);
        } else {
            v.S = (i128)a;
        }
    }
    Agg total;
    const Agg ex = block_exclusive_scan(v, total);
    if (i < n) {
        const Agg base = tiles[blockIdx.x];
        const int32_t light_rank = base.lights + ex.lights;
        if (a < 0) {
            lights[light_rank] = (int32_t)i;
            Dexcl[light_rank] = base.D + ex.D;
        } else {
            const int32_t heavy_rank = (int32_t)i - light_rank;
            heavies[heavy_rank] = (int32_t)i;
            Sincl[heavy_rank] = base.S + ex.S + v.S;
        }
    }
}

__device__ __forceinline__ float pdf_of(long long m, unsigned long long W) { return (float)((double)m / (double)W); }

// (float)(x / Wd) for a whole x >= 0, with inv = 1 / Wd: the product x inv is
// within two units of the last place of the quotient, so both round to the same
// float unless the product's 29 bits below a float's lie that close to half; there
// (once in 2^26) the division decides. FP64 runs at 1/64 of the FP32 rate, and a
// division is some ten operations. Below 2^-126, where a float has fewer bits, the
// division decides as well, but not for 0, the weight of everything that does not
// emit (66,356 weights, 2 % / 98 % of them 0: 28.8 -> 27.2 / 30.1 -> 29.2 us).
__device__ __forceinline__ float ratio_f(double x, double Wd, double inv)
{
    const double q = x * inv;
    const uint32_t low = (uint32_t)__double2loint(q) & 0x1fffffffu, high = (uint32_t)__double2hiint(q);
    // high - 1 of a zero wraps round; 2^-126 has the high word (1023 - 126) << 20
    if (low - 0x0ffffffcu <= 8u || high - 1u < ((1023u - 126u) << 20) - 1u) return (float)(x / Wd);
    return (float)q;
}

// First index of the sorted list with list[i] > key (Greater) or >= key, as a
// binary search that starts from every (count / 256)-th entry, staged in shared
// memory.
constexpr int kCoarse = 256;
template <bool GREATER>
__device__ __forceinline__ int32_t list_search(const i128 *list, int32_t count, const i128 *coarse, int32_t step, i128 key)
{
    // coarse[c] = list[min((c + 1) step, count) - 1]
    int32_t lo = 0, hi = kCoarse;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (GREATER ? coarse[mid] > key : coarse[mid] >= key) hi = mid;
        else lo = mid + 1;
    }
    if (lo == kCoarse) return count;
    hi = min((lo + 1) * step, count) - 1;  // satisfies the condition
    lo = lo * step;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (GREATER ? list[mid] > key : list[mid] >= key) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// The entry of list item t (the lights in order, then the heavies); s_S and s_D
// are the staged entries of list_search.
__device__ __forceinline__ void sweep_assign_item(uint32_t t, const float *__restrict__ w, uint32_t n, const SweepScalars &s,
                                                  const int32_t *lights, const i128 *Dexcl, const int32_t *heavies,
                                                  const i128 *Sincl, const i128 *s_S, int32_t step_S, const i128 *s_D,
                                                  int32_t step_D, dr_alias_entry *__restrict__ out)
{
    const int32_t nl = s.num_lights, nh = s.num_heavies;
    const double Wd = s.Wd, inv = s.inv_W;
    auto fixed_d = [&](int32_t i) { return fixed_weight_double(clamp_weight(w[i]), s.shift); };
    auto pdf = [&](int32_t i) { return ratio_f(fixed_d(i), Wd, inv); };
    dr_alias_entry e;
    int32_t slot;
    if ((int32_t)t < nl) {
        const int32_t k = (int32_t)t;
        const int32_t i = lights[k];
        slot = i;
        const double m = fixed_d(i);
        // first heavy h with Sincl[h] > d
        const int32_t h = nh > 0 ? list_search<true>(Sincl, nh, s_S, step_S, Dexcl[k]) : 0;
        e.A = i;
        e.p_A = ratio_f(m * s.nd, Wd, inv);  // n m, rounded to a double once
        e.pdf_A = ratio_f(m, Wd, inv);
        if (h < nh) {
            e.B = heavies[h];
            e.pdf_B = pdf(e.B);
        } else {
            e.B = -1;
            e.pdf_B = 0.0f;
            e.p_A = 1.0f;
        }
    } else {
        const int32_t j = (int32_t)t - nl;
        const int32_t i = heavies[j];
        slot = i;
        const i128 sj = Sincl[j];
        // first light k with Dexcl[k] >= Sincl[j]
        const int32_t k = nl > 0 ? list_search<false>(Dexcl, nl, s_D, step_D, sj) : 0;
        const i128 Dk = k < nl ? Dexcl[k] : s.D_total;
        const long long R = (long long)(sj - Dk);
        e.A = i;
        e.pdf_A = pdf(i);
        if (j + 1 < nh) {
            e.p_A = ratio_f((double)((long long)s.W + R), Wd, inv);
            e.B = heavies[j + 1];
            e.pdf_B = pdf(e.B);
        } else {
            e.p_A = 1.0f;
            e.B = -1;
            e.pdf_B = 0.0f;
        }
        if (e.p_A == 1.0f) {
            e.B = -1;
            e.pdf_B = 0.0f;
        }
    }
    ensure_pa_larger(e);
    out[slot] = e;
}

__device__ __forceinline__ int32_t coarse_step(int32_t count) { return (count + kCoarse - 1) / kCoarse; }

__global__ void __launch_bounds__(kCoarse) k_sweep_assign(const float *__restrict__ w, uint32_t n, const SweepScalars *sc,
                                                          const int32_t *lights, const i128 *Dexcl, const int32_t *heavies,
                                                          const i128 *Sincl, dr_alias_entry *__restrict__ out)
{
    // the lists may still be written when this kernel is launched, so they are
    // not read through the read-only path
    wait_previous();
    const SweepScalars s = *sc;
    const uint32_t t = blockIdx.x * kCoarse + threadIdx.x;
    if (s.uniform) {
        if (t < n) out[t] = dr_alias_entry{1.0f, 1.0f / (float)n, 0.0f, (int32_t)t, -1};
        return;
    }
    const int32_t nl = s.num_lights, nh = s.num_heavies;
    // blocks of lights search the heavies and blocks of heavies the lights; the
    // one that holds both stages both
    __shared__ i128 s_S[kCoarse], s_D[kCoarse];
    const int32_t step_S = coarse_step(nh), step_D = coarse_step(nl), begin = (int32_t)(blockIdx.x * kCoarse);
    if (begin < nl && nh > 0) s_S[threadIdx.x] = Sincl[min((int32_t)(threadIdx.x + 1) * step_S, nh) - 1];
    if (begin + kCoarse > nl && nl > 0) s_D[threadIdx.x] = Dexcl[min((int32_t)(threadIdx.x + 1) * step_D, nl) - 1];
    __syncthreads();
    if (t < n) sweep_assign_item(t, w, n, s, lights, Dexcl, heavies, Sincl, s_S, step_S, s_D, step_D, out);
}

// ---- sweep build of one table by one cluster of blocks ---------------------------------

// The first six steps of the parallel build (scalars, exponent, total, tile
// sums, their scan, the lists) as one launch: every thread keeps up to kListItems
// consecutive items in registers, and the blocks of one cluster meet through
// distributed shared memory. The same integers in the same order as the separate
// kernels, without their launches and re-reads; bound by the latency of its four
// meetings and of the scattered list stores. Build of 66,356 weights 42.5 ->
// 29 us, of 1,000 33 -> 17 us, of 3 28 -> 13 us; 131,072 weights 57 -> 39 us (the
// separate kernels, which take over above, 53 us at 131,073).
constexpr int kListBlock = 1024, kListItems = 8;
constexpr unsigned kListCluster = 16;
// Tables of up to this many weights get their entries from the same launch
// (100 weights: 16.8 -> 14.0 us; at 1,000 one SM's FP64 units take longer than
// another launch: 16.8 -> 25.0 us).
constexpr uint32_t kListWhole = 256;
static_assert(kListWhole <= kListBlock, "one block");

__global__ void __launch_bounds__(kListBlock) k_sweep_lists(const float *__restrict__ w, uint32_t n, uint32_t per_thread,
                                                            SweepScalars *sc, int32_t *lights, i128 *Dexcl, int32_t *heavies,
                                                            i128 *Sincl, dr_alias_entry *__restrict__ out)
{
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank(), blocks = cluster.num_blocks();
    struct Meet {
        int emax;
        unsigned long long W;
        int lights;
        i128 D, S;
    };
    __shared__ Meet s_meet;  // this block's sums, read by the others
    __shared__ Meet s_all;   // over the cluster (exponent, total), or over the blocks before this one
    __shared__ int s_all_lights;
    __shared__ i128 s_all_D;
    __shared__ unsigned long long s_warp[32];
    __shared__ int s_cnt[32];
    __shared__ i128 s_D[32], s_S[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = (rank * kListBlock + threadIdx.x) * per_thread;
    allow_next();
    float x[kListItems];
    int e = INT_MIN;
#pragma unroll
    for (int k = 0; k < kListItems; ++k) {
        x[k] = (uint32_t)k < per_thread && first + k < n ? clamp_weight(w[first + k]) : 0.0f;
        if (x[k] > 0.0f) e = max(e, float_exponent(x[k]));
    }
    // largest exponent: of the block, then one lane per block of the cluster
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) s_cnt[warp] = e;
    __syncthreads();
    if (warp == 0) {
        e = __reduce_max_sync(0xffffffffu, s_cnt[lane]);
        if (lane == 0) s_meet.emax = e;
    }
    cluster.sync();
    if (warp == 0) {
        e = (unsigned)lane < blocks ? cluster.map_shared_rank(&s_meet, lane)->emax : INT_MIN;
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) s_all.emax = e;
    }
    __syncthreads();
    e = s_all.emax;
    const int lg = 32 - __clz((int)n);  // smallest lg with 2^lg >= n + 1
    const int shift = 61 - lg - e;
    // total
    auto weight_of = [&](int k) { return e == INT_MIN ? 0ll : fixed_weight_bits(x[k], shift); };
    unsigned long long W = 0;
#pragma unroll
    for (int k = 0; k < kListItems; ++k) W += (unsigned long long)weight_of(k);
    for (int off = 16; off > 0; off >>= 1) W += __shfl_xor_sync(0xffffffffu, W, off);
    if (lane == 0) s_warp[warp] = W;
    __syncthreads();
    if (warp == 0) {
        W = s_warp[lane];
        for (int off = 16; off > 0; off >>= 1) W += __shfl_xor_sync(0xffffffffu, W, off);
        if (lane == 0) s_meet.W = W;
    }
    cluster.sync();
    if (warp == 0) {
        W = (unsigned)lane < blocks ? cluster.map_shared_rank(&s_meet, lane)->W : 0ull;
        for (int off = 16; off > 0; off >>= 1) W += __shfl_xor_sync(0xffffffffu, W, off);
        if (lane == 0) s_all.W = W;
    }
    __syncthreads();
    W = s_all.W;
    // light count, deficit and surplus sums before each thread's items
    int cnt = 0;
    i128 D = 0, S = 0;
#pragma unroll
    for (int k = 0; k < kListItems; ++k) {
        if ((uint32_t)k >= per_thread || first + k >= n) break;
        const long long a = (long long)n * weight_of(k) - (long long)W;
        if (a < 0) {
            ++cnt;
            D += (i128)(-a);
        } else {
            S += (i128)a;
        }
    }
    const int c_inc = warp_scan_int(cnt);
    const i128 d_inc = warp_scan_i128(D), s_inc = warp_scan_i128(S);
    if (lane == 31) s_cnt[warp] = c_inc, s_D[warp] = d_inc, s_S[warp] = s_inc;
    __syncthreads();
    if (warp == 0) {
        const int c = warp_scan_int(s_cnt[lane]);
        const i128 d = warp_scan_i128(s_D[lane]), q = warp_scan_i128(s_S[lane]);
        s_cnt[lane] = c, s_D[lane] = d, s_S[lane] = q;
        if (lane == 31) s_meet.lights = c, s_meet.D = d, s_meet.S = q;
    }
    cluster.sync();
    if (warp == 0) {
        int c = 0;
        i128 d = 0, q = 0;
        if ((unsigned)lane < blocks) {
            const Meet *o = cluster.map_shared_rank(&s_meet, lane);
            c = o->lights, d = o->D, q = o->S;
        }
        const int ci = warp_scan_int(c);
        const i128 di = warp_scan_i128(d), qi = warp_scan_i128(q);
        if ((unsigned)lane == rank) s_all.lights = ci - c, s_all.D = di - d, s_all.S = qi - q;
        if (lane == 31) s_all_lights = ci, s_all_D = di;
    }
    cluster.sync();  // no block leaves while another reads its sums
    int rank_l = s_all.lights + c_inc - cnt + (warp > 0 ? s_cnt[warp - 1] : 0);
    i128 Db = s_all.D + d_inc - D + (warp > 0 ? s_D[warp - 1] : (i128)0);
    i128 Sb = s_all.S + s_inc - S + (warp > 0 ? s_S[warp - 1] : (i128)0);
    // the lists, in index order, with their running sums
#pragma unroll
    for (int k = 0; k < kListItems; ++k) {
        if ((uint32_t)k >= per_thread || first + k >= n) break;
        const long long a = (long long)n * weight_of(k) - (long long)W;
        if (a < 0) {
            lights[rank_l] = (int32_t)(first + k);
            Dexcl[rank_l] = Db;
            ++rank_l;
            Db += (i128)(-a);
        } else {
            const int32_t h = (int32_t)(first + k) - rank_l;
            Sb += (i128)a;
            heavies[h] = (int32_t)(first + k);
            Sincl[h] = Sb;
        }
    }
    __shared__ SweepScalars s_sc;
    if (threadIdx.x == 0) {
        const float Wf = e == INT_MIN ? 0.0f : (float)ldexp((double)W, -shift);
        s_sc.emax = e;
        s_sc.lg = lg;
        s_sc.shift = shift;
        s_sc.uniform = !(Wf >= 1e-5f);
        s_sc.W = W;
        s_sc.num_lights = s_all_lights;
        s_sc.num_heavies = (int32_t)n - s_all_lights;
        s_sc.D_total = s_all_D;
        s_sc.Wd = (double)W;
        s_sc.inv_W = 1.0 / s_sc.Wd;
        s_sc.nd = (double)n;
        if (rank == 0) *sc = s_sc;
    }
    if (n > kListWhole) return;
    // a small table's entries too, without another launch
    __shared__ i128 s_fine_S[kCoarse], s_fine_D[kCoarse];
    __syncthreads();
    const SweepScalars &s = s_sc;
    const int32_t step_S = coarse_step(s.num_heavies), step_D = coarse_step(s.num_lights), c = (int32_t)threadIdx.x;
    if (c < kCoarse && s.num_heavies > 0) s_fine_S[c] = Sincl[min((c + 1) * step_S, s.num_heavies) - 1];
    if (c < kCoarse && s.num_lights > 0) s_fine_D[c] = Dexcl[min((c + 1) * step_D, s.num_lights) - 1];
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < n; t += kListBlock) {
        if (s.uniform) out[t] = dr_alias_entry{1.0f, 1.0f / (float)n, 0.0f, (int32_t)t, -1};
        else sweep_assign_item(t, w, n, s, lights, Dexcl, heavies, Sincl, s_fine_S, step_S, s_fine_D, step_D, out);
    }
}

// The launch of one cluster of `blocks` blocks.
struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    ClusterLaunch(unsigned blocks, cudaStream_t st)
    {
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(kListBlock);
        cfg.stream = st;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = blocks;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// The largest cluster of k_sweep_lists that the current device can run: 16
// blocks, more than the 8 that every device offers, need as many free SMs in one
// of its SM clusters, which a partition of a GPU may not have. 0: none.
static unsigned list_cluster_limit()
{
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static int known[kMaxDevices];  // limit + 1
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (known[device] == 0) {
        unsigned limit = kListCluster;
        if (cudaFuncSetAttribute(k_sweep_lists, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) limit = 8;
        for (; limit > 0; limit /= 2) {
            const ClusterLaunch l(limit, nullptr);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k_sweep_lists, &l.cfg) == cudaSuccess && clusters > 0) break;
        }
        cudaGetLastError();
        known[device] = (int)limit + 1;
    }
    return (unsigned)known[device] - 1;
}

static cudaError_t launch_sweep_lists(const float *w, uint32_t n, unsigned max_blocks, SweepScalars *sc, int32_t *lights, i128 *Dexcl,
                                      int32_t *heavies, i128 *Sincl, dr_alias_entry *out, cudaStream_t st)
{
    // as few blocks as give every thread one item, up to the largest cluster; then more items
    unsigned blocks = 1;
    while (blocks < max_blocks && (uint64_t)blocks * kListBlock < n) blocks *= 2;
    const uint32_t per_thread = (n + blocks * kListBlock - 1) / (blocks * kListBlock);
    const ClusterLaunch l(blocks, st);
    const cudaError_t e = cudaLaunchKernelEx(&l.cfg, k_sweep_lists, w, n, per_thread, sc, lights, Dexcl, heavies, Sincl, out);
    if (e != cudaSuccess || n <= kListWhole) return e;
    return launch_after(k_sweep_assign, (n + kCoarse - 1) / kCoarse, kCoarse, 0, st, w, n, sc, lights, Dexcl, heavies, Sincl, out);
}

// ---- sweep build of many small tables, one thread per table ---------------------------

// The sweep build of one table by one thread: the same fixed-point quantities
// (m_i, W, a_i = n m_i - W) as the parallel kernels above and the same
// assignment rules, evaluated by two cursors that walk the lights and the
// heavies in index order instead of prefix sums and binary searches. O(n), no
// scratch memory; the table equals the parallel build's bit for bit.
__device__ void alias_sweep_build_one(const float *__restrict__ w, uint32_t n, dr_alias_entry *__restrict__ out)
{
    if (n == 0) return;
    SweepScalars s;
    s.emax = INT_MIN;
    for (uint32_t i = 0; i < n; ++i) {
        const float x = clamp_weight(w[i]);
        if (x > 0.0f) s.emax = max(s.emax, float_exponent(x));
    }
    int lg = 0;
    while ((1ll << lg) < (long long)n + 1) ++lg;
    s.lg = lg;
    s.shift = 61 - lg - s.emax;
    unsigned long long W = 0;
    for (uint32_t i = 0; i < n; ++i) W += (unsigned long long)fixed_weight(w[i], s);
    const float Wf = s.emax == INT_MIN ? 0.0f : (float)ldexp((double)W, -s.shift);
    if (!(Wf >= 1e-5f)) {
        const float u = 1.0f / (float)n;
        for (uint32_t i = 0; i < n; ++i) out[i] = dr_alias_entry{1.0f, u, 0.0f, (int32_t)i, -1};
        return;
    }
    const double Wd = (double)W;
    const long long nn = (long long)n;
    auto surplus = [&](uint32_t i) { return nn * fixed_weight(w[i], s) - (long long)W; };  // a_i
    auto next_heavy = [&](uint32_t i) {
        while (i < n && surplus(i) < 0) ++i;
        return i;
    };
    auto next_light = [&](uint32_t i) {
        while (i < n && surplus(i) >= 0) ++i;
        return i;
    };
    // lights: alias = first heavy h whose inclusive surplus sum exceeds the
    // deficits of the lights before this one
    {
        uint32_t h = next_heavy(0);
        i128 S = h < n ? (i128)surplus(h) : (i128)0;
        i128 D = 0;
        for (uint32_t i = next_light(0); i < n; i = next_light(i + 1)) {
            while (h < n && !(S > D)) {
                h = next_heavy(h + 1);
                if (h < n) S += (i128)surplus(h);
            }
            const long long m = fixed_weight(w[i], s);
            dr_alias_entry e;
            e.A = (int32_t)i;
            e.p_A = (float)((double)(nn * m) / Wd);
            e.pdf_A = pdf_of(m, W);
            if (h < n) {
                e.B = (int32_t)h;
                e.pdf_B = pdf_of(fixed_weight(w[h], s), W);
            } else {
                e.B = -1;
                e.pdf_B = 0.0f;
                e.p_A = 1.0f;
            }
            ensure_pa_larger(e);
            out[i] = e;
            D += (i128)(-surplus(i));
        }
    }
    // heavies: R = inclusive surplus sum - deficits of the lights before the
    // first light not covered by it; alias = the next heavy
    {
        uint32_t k = next_light(0);
        i128 Dk = 0, S = 0;
        for (uint32_t j = next_heavy(0); j < n;) {
            S += (i128)surplus(j);
            while (k < n && !(Dk >= S)) {
                Dk += (i128)(-surplus(k));
                k = next_light(k + 1);
            }
            const long long R = (long long)(S - Dk);
            const uint32_t jn = next_heavy(j + 1);
            dr_alias_entry e;
            e.A = (int32_t)j;
            e.pdf_A = pdf_of(fixed_weight(w[j], s), W);
            if (jn < n) {
                e.p_A = (float)((double)((long long)W + R) / Wd);
                e.B = (int32_t)jn;
                e.pdf_B = pdf_of(fixed_weight(w[jn], s), W);
            } else {
                e.p_A = 1.0f;
                e.B = -1;
                e.pdf_B = 0.0f;
            }
            if (e.p_A == 1.0f) {
                e.B = -1;
                e.pdf_B = 0.0f;
            }
            ensure_pa_larger(e);
            out[j] = e;
            j = jn;
        }
    }
}

// Many independent sweep tables, one thread each (segments as k_alias_ref_segments).
__global__ void k_alias_sweep_segments(const float *__restrict__ w, const uint32_t *__restrict__ begin,
                                       const uint32_t *__restrict__ count, uint32_t nseg,
                                       dr_alias_entry *__restrict__ out)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    const uint32_t b = begin[s];
    alias_sweep_build_one(w + b, count[s], out + b);
}

// ---- sampling ------------------------------------------------------------------------------

// sample() (include/tracing/DistributionSamplers.hpp:64-88) with the two
// uniforms of draw i at uniforms[2i], uniforms[2i+1].
__global__ void k_alias_sample(const dr_alias_entry *__restrict__ table, uint32_t n, const float *__restrict__ u,
                               uint64_t draws, int32_t *__restrict__ index, float *__restrict__ pdf)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= draws) return;
    const float2 r = reinterpret_cast<const float2 *>(u)[i];
    int32_t idx;
    float p;
    alias_sample(table, n, r.x, r.y, idx, p);
    index[i] = idx;
    pdf[i] = p;
}

// ---- launchers -------------------------------------------------------------------------------

size_t alias_scratch_bytes(uint32_t n, int mode)
{
    if (mode == DR_ALIAS_REFERENCE) return 256 + (size_t)n * (8 + 8 + 4) + 64;
    const size_t tiles = (n + kSweepBlock - 1) / kSweepBlock;
    return 512 + tiles * sizeof(Agg) + (size_t)n * (4 + 4 + 16 + 16) + 256;
}

static inline char *align256(char *p) { return reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255)); }

cudaError_t launch_alias_build(const float *w, uint32_t n, dr_alias_entry *out, int mode, void *scratch,
                               size_t scratch_bytes, int num_sms, cudaStream_t st, unsigned max_cluster)
{
    if (n == 0) return cudaSuccess;
    if (scratch_bytes < alias_scratch_bytes(n, mode)) return cudaErrorInvalidValue;
    char *p = align256(static_cast<char *>(scratch));
    if (mode == DR_ALIAS_REFERENCE) {
        float *total = reinterpret_cast<float *>(p);
        p = align256(p + 16);
        HeapItem *under = reinterpret_cast<HeapItem *>(p);
        HeapItem *over = under + n;
        float *filtered = reinterpret_cast<float *>(over + n);
        k_alias_ref_pair<<<1, 32, 0, st>>>(w, n, out, under, over, filtered, total);
        const int blocks = (int)std::min<uint32_t>((n + 255) / 256, (uint32_t)num_sms * 4);
        k_alias_ref_pdfs<<<blocks, 256, 0, st>>>(n, out, filtered, total);
        return cudaGetLastError();
    }
    SweepScalars *sc = reinterpret_cast<SweepScalars *>(p);
    p = align256(p + sizeof(SweepScalars));
    const uint32_t tiles = (n + kSweepBlock - 1) / kSweepBlock;
    Agg *tile_agg = reinterpret_cast<Agg *>(p);
    p = align256(p + tiles * sizeof(Agg));
    i128 *Dexcl = reinterpret_cast<i128 *>(p);
    i128 *Sincl = Dexcl + n;
    int32_t *lights = reinterpret_cast<int32_t *>(Sincl + n);
    int32_t *heavies = lights + n;
    // the one-launch lists up to 8 items per thread of a cluster: 131,072 weights with 16 blocks
    const unsigned cluster = std::min(list_cluster_limit(), max_cluster);
    if (n <= (uint64_t)cluster * kListBlock * kListItems)
        return launch_sweep_lists(w, n, cluster, sc, lights, Dexcl, heavies, Sincl, out, st);
    const int grid = (int)std::min<uint32_t>((n + 255) / 256, (uint32_t)num_sms * 8);
    k_sweep_init<<<1, 32, 0, st>>>(sc, n);
    k_sweep_exponent<<<grid, 256, 0, st>>>(w, n, sc);
    k_sweep_sum<<<grid, 256, 0, st>>>(w, n, sc);
    k_sweep_tile_aggregates<<<tiles, kSweepBlock, 0, st>>>(w, n, sc, tile_agg);
    k_sweep_scan_tiles<<<1, kSweepBlock, 0, st>>>(tile_agg, tiles, sc, n);
    k_sweep_scatter<<<tiles, kSweepBlock, 0, st>>>(w, n, sc, tile_agg, lights, Dexcl, heavies, Sincl);
    k_sweep_assign<<<(n + kCoarse - 1) / kCoarse, kCoarse, 0, st>>>(w, n, sc, lights, Dexcl, heavies, Sincl, out);
    return cudaGetLastError();
}

cudaError_t launch_alias_ref_segments(const float *w, uint32_t total_n, const uint32_t *begin, const uint32_t *count,
                                     uint32_t nseg, dr_alias_entry *out, void *scratch, size_t scratch_bytes,
                                     cudaStream_t st)
{
    if (nseg == 0) return cudaSuccess;
    if (scratch_bytes < (size_t)total_n * (2 * sizeof(HeapItem) + sizeof(float)) + 512) return cudaErrorInvalidValue;
    char *p = align256(static_cast<char *>(scratch));
    HeapItem *heaps = reinterpret_cast<HeapItem *>(p);
    float *filtered = reinterpret_cast<float *>(heaps + 2 * (size_t)total_n);
    k_alias_ref_segments<<<(nseg + 63) / 64, 64, 0, st>>>(w, begin, count, nseg, out, heaps, filtered);
    return cudaGetLastError();
}

cudaError_t launch_alias_sweep_segments(const float *w, const uint32_t *begin, const uint32_t *count, uint32_t nseg,
                                       dr_alias_entry *out, cudaStream_t st)
{
    if (nseg == 0) return cudaSuccess;
    k_alias_sweep_segments<<<(nseg + 63) / 64, 64, 0, st>>>(w, begin, count, nseg, out);
    return cudaGetLastError();
}

cudaError_t launch_alias_sample(const dr_alias_entry *table, uint32_t n, const float *u, uint64_t draws,
                                int32_t *index, float *pdf, cudaStream_t st)
{
    if (draws == 0) return cudaSuccess;
    const uint64_t blocks = (draws + 255) / 256;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    k_alias_sample<<<(unsigned)blocks, 256, 0, st>>>(table, n, u, draws, index, pdf);
    return cudaGetLastError();
}

}  // namespace dr
