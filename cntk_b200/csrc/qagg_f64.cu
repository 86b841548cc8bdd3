// qagg_f64.cu -- the column quantizer for ElemType = double: 64-bit packed words (QuantizedWordHelper<double>::ValueType,
// Source/Math/ValueQuantizer.h:48-55), 64 one-bit values per word, bit widths 1 .. 64.  This is what the reference's own
// 1-bit end-to-end tests run (precision=double).  Single-matrix entry points only (MatrixQuantizerImpl<double>); the
// striped aggregator is built for float.
//
// Same arithmetic contract as the float kernels: every operation an explicit round-to-nearest double intrinsic, operand
// types as the reference's (size_t -> double before divides, unsigned x double, truncating double -> int64), the float
// literals 1e-36f / 0.5f / 2.0f / 4.0f promoted as the reference's template does, and every per-column sum accumulated in
// ROW ORDER.  A column's walk is a chain of M dependent double adds per level, so everything else is arranged around
// having that chain run undisturbed: one CTA per column; all threads stage v = gradient + residual in shared memory and count
// the rows below a threshold of 0; then lane 0 of warp 0 walks the lower level (or the single sum of the other modes) and
// lane 0 of warp 1 the upper one, the next eight rows always loaded ahead of the adds; then all threads quantize.  The columns
// an SM holds are the chains it keeps going, so the CTA's size follows the number of columns (launch_shape_d).
#include "../../include/qagg.h"
#include "qagg_internal.h"

#include <algorithm>

namespace qagg {

// Two forms of the quantize kernel.  FEW: eight warps and as many rows in shared memory as help, for matrices whose columns all
// have a CTA at once even so.  MANY: four warps of at most 32 registers and short chunks, 16 CTAs per SM.
constexpr int DFEW_THREADS = 256, DFEW_CTAS = 5;
constexpr int DMANY_THREADS = 128, DMANY_CTAS = 16;
constexpr int DFEW_RESIDENT = 24576; // most rows of a column that stays in shared memory (192 KB)
constexpr int DFEW_CHUNK = 4096;     // rows per staged chunk of one that does not
constexpr int DFEW_TASKS = 1024;     // most pieces of words (see `split`) of a column
constexpr int DMANY_CHUNK = 1024;    // (1536 rows fit too, but leave less L1 for the second read: 9304 x 2048 at 8 bits 220 -> 250 us)

struct ValQD
{
    double qmin, qmax, qmid, qfactor, ufactor;
    unsigned long long rangeend;
};

// ValueQuantizer<double> constructor (ValueQuantizer.h:68-97)
__device__ __forceinline__ ValQD make_valq_d(int bits, double lower, double upper)
{
    ValQD q;
    q.qmin = lower;
    q.qmax = upper;
    q.rangeend = (bits >= 64) ? 0ull : (1ull << bits);
    const double range = __dsub_rn(upper, lower);
    if ((range < (double) 1e-36f) || (q.rangeend == 0))
    {
        q.qfactor = q.ufactor = 0.0;
    }
    else
    {
        const double used = (double) (q.rangeend - (bits > 1 ? 1ull : 0ull)); // size_t -> double
        q.qfactor = __ddiv_rn(used, range);
        q.ufactor = __ddiv_rn(range, used);
    }
    q.qmid = __dmul_rn((double) 0.5f, __dadd_rn(upper, lower));
    return q;
}

// Quantize<ZeroThresholdFor1Bit> (ValueQuantizer.h:101-128, 144-156) for more than one bit
__device__ __forceinline__ unsigned long long quantize_d(const ValQD& q, int bits, double u)
{
    if (bits == 64)
        return (unsigned long long) __double_as_longlong(u);
    if (u <= q.qmin)
        return 0ull;
    if (u >= q.qmax)
        return q.rangeend - 1ull;
    return (unsigned long long) __double2ll_rz(__dmul_rn(__dsub_rn(u, q.qmin), q.qfactor));
}

// Unquantize (ValueQuantizer.h:131-141)
__device__ __forceinline__ double unquantize_d(const ValQD& q, int bits, unsigned long long u)
{
    if (bits == 64)
        return __longlong_as_double((long long) u);
    return __dadd_rn(__dmul_rn(__dadd_rn(__ull2double_rn(u), 0.5), q.ufactor), q.qmin);
}

enum
{
    DWALK_SUM = 0, // acc += v
    DWALK_SQUARES, // acc += v * v
    DWALK_BELOW,   // acc += v where v < threshold (every other row adds +0: the sum starts at +0 and stays exact)
    DWALK_REST     // acc += v in all other rows (a NaN lands here, as in the reference)
};
template <int KIND>
__device__ __forceinline__ double dwalk_term(double v, double threshold)
{
    if (KIND == DWALK_SQUARES)
        return __dmul_rn(v, v);
    if (KIND == DWALK_BELOW)
        return (v < threshold) ? v : 0.0;
    if (KIND == DWALK_REST)
        return (v < threshold) ? 0.0 : v;
    return v;
}
// one lane, rows in order; eight rows per trip with the next eight already loaded (the prefetch of the last trip is clamped)
template <int KIND>
__device__ __forceinline__ double dwalk(const double* __restrict__ sv, int nr, double acc, double threshold)
{
    const int trips = nr >> 3;
    const double2* const p = reinterpret_cast<const double2*>(sv);
    if (trips > 0)
    {
        double2 a[4], n[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            a[i] = p[i];
        for (int t = 0; t < trips; ++t)
        {
            const int nx = (t + 1 < trips ? t + 1 : t) * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                n[i] = p[nx + i];
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                acc = __dadd_rn(acc, dwalk_term<KIND>(a[i].x, threshold));
                acc = __dadd_rn(acc, dwalk_term<KIND>(a[i].y, threshold));
                a[i] = n[i];
            }
        }
    }
    for (int i = trips << 3; i < nr; ++i)
        acc = __dadd_rn(acc, dwalk_term<KIND>(sv[i], threshold));
    return acc;
}

// stages rows [r0, r0 + nr) of v = gradient + residual and, with COUNT, returns how many of this thread's rows are below `threshold`
template <bool COUNT>
__device__ __forceinline__ unsigned dstage(double* __restrict__ sv, const double* __restrict__ g, const double* r, int nr, double threshold)
{
    unsigned below = 0;
#pragma unroll 4
    for (int i = threadIdx.x; i < nr; i += blockDim.x)
    {
        const double v = __dadd_rn(g[i], r[i]);
        sv[i] = v;
        if (COUNT)
            below += (v < threshold) ? 1u : 0u;
    }
    return below;
}

// ComputeRangeStatColjSubset for one column (ColumnQuantizer.h:209-341) + Quantize (ColumnQuantizer.h:50-65, 90-147).
// `chunk` rows are staged at a time; a column of up to `chunk` rows is read from memory once and stays for the quantization.
// `split` threads share a packed word.  Word w holds rows w, w + Q, ...: with few words (a 512-row column has 8 at 1 bit) one
// thread per word would leave the CTA idle, so each of the `split` threads takes every split-th row of the word and ORs its fields
// in shared memory; task t = (t / Q, t % Q) then covers rows t, t + split * Q, ...: neighbouring threads, neighbouring rows.
// `pair`: two staging buffers that take turns, so that a warp that is done with a column goes on to load the next one.
template <int THREADS, int CTAS, bool ONEBIT>
__global__ void __launch_bounds__(THREADS, CTAS) k_quantize_f64(const double* __restrict__ grad, const double* resIn, double* resOut,
                                                               unsigned char* __restrict__ packed, int M, unsigned N, int bits, int zeroThr, int chunk,
                                                               int split, int pair)
{
    extern __shared__ __align__(16) double smem[];
    __shared__ double sAcc[2];
    __shared__ unsigned sNum0;
    __shared__ ValQD sQ;         // the column's quantizer: divided out once, not by every thread
    __shared__ double sLevel[2]; // 1 bit: what the two values unquantize to
    const int tid = threadIdx.x, nt = blockDim.x;
    const int Q = (int) (((long long) M * bits + 63) / 64); // M < 2^30, so with 64 bits Q = M still fits
    const int svStride = (chunk + 1) & ~1;
    unsigned* const sWords = reinterpret_cast<unsigned*>(smem + svStride); // split > 1: the column's words as 2 Q halves
    double* sv = smem;
    const bool resident = M <= chunk;
    const int tasks = Q * split;
    // the count and the words are zero whenever a column begins: whoever consumes them clears them
    if (tid == 0)
        sNum0 = 0u;
    if (split > 1)
        for (int w = tid; w < 2 * Q; w += nt)
            sWords[w] = 0u;
    __syncthreads();
    for (unsigned j = blockIdx.x; j < N; j += gridDim.x)
    {
        const double* __restrict__ g = grad + (long long) j * M;
        const double* r = resIn + (long long) j * M;
        double mean = 0.0;
        // mean-threshold 1-bit mode: a first ordered pass for the column mean (:232-245)
        if (ONEBIT && !zeroThr)
        {
            double acc = 0.0;
            for (int r0 = 0; r0 < M; r0 += chunk)
            {
                const int nr = min(chunk, M - r0);
                dstage<false>(sv, g + r0, r + r0, nr, 0.0);
                __syncthreads();
                if (tid == 0)
                    acc = dwalk<DWALK_SUM>(sv, nr, acc, 0.0);
                __syncthreads();
            }
            if (tid == 0)
                sAcc[0] = __ddiv_rn(acc, (double) (unsigned long long) M); // size_t -> double
            __syncthreads();
            mean = sAcc[0];
        }
        // the ordered sums: two level sums and a count (1 bit), or the sum of squares (otherwise)
        double acc = 0.0;
        for (int r0 = 0; r0 < M; r0 += chunk)
        {
            const int nr = min(chunk, M - r0);
            if (ONEBIT)
            {
                unsigned below = 0;
                if (resident && !zeroThr) // already staged
                    for (int i = tid; i < nr; i += nt)
                        below += (sv[i] < mean) ? 1u : 0u;
                else
                    below = dstage<true>(sv, g + r0, r + r0, nr, mean);
                below = __reduce_add_sync(0xffffffffu, below);
                if ((tid & 31) == 0 && below)
                    atomicAdd(&sNum0, below);
            }
            else
            {
                dstage<false>(sv, g + r0, r + r0, nr, 0.0);
            }
            __syncthreads();
            if (!ONEBIT)
            {
                if (tid == 0)
                    acc = dwalk<DWALK_SQUARES>(sv, nr, acc, 0.0);
            }
            else if (tid == 0)
            {
                acc = dwalk<DWALK_BELOW>(sv, nr, acc, mean);
            }
            else if (tid == 32)
            {
                acc = dwalk<DWALK_REST>(sv, nr, acc, mean);
            }
            if (!resident)
                __syncthreads();
        }
        if (ONEBIT)
        {
            if (tid == 32)
                sAcc[1] = acc;
            __syncthreads();
        }
        unsigned char* const colp = packed + (long long) j * (16 + 8 * (long long) Q);
        if (tid == 0)
        {
            const double rows = (double) (unsigned long long) M; // size_t -> double
            double lower, upper;
            if (ONEBIT)
            {
                unsigned n0 = sNum0, n1 = (unsigned) M - n0;
                sNum0 = 0u;
                const double a0 = acc, a1 = sAcc[1];
                double radius, newmean;
                if (!zeroThr)
                {
                    const double devacc0 = __dsub_rn(__dmul_rn((double) n0, mean), a0);
                    const double devacc1 = __dsub_rn(a1, __dmul_rn((double) n1, mean));
                    const double dev = __ddiv_rn(__dadd_rn(devacc0, devacc1), rows);
                    radius = __dmul_rn((double) 2.0f, dev);
                    newmean = mean;
                }
                else
                {
                    if (n0 == 0)
                        n0 = 1;
                    if (n1 == 0)
                        n1 = 1;
                    const double mean0 = __ddiv_rn(a0, (double) n0);
                    const double mean1 = __ddiv_rn(a1, (double) n1);
                    newmean = __dmul_rn((double) 0.5f, __dadd_rn(mean0, mean1));
                    radius = __dmul_rn((double) 2.0f, __dsub_rn(mean1, newmean));
                }
                lower = __dsub_rn(newmean, radius);
                upper = __dadd_rn(newmean, radius);
            }
            else
            {
                const double stddev = __dsqrt_rn(__ddiv_rn(acc, rows));
                const double w = __dmul_rn((double) 4.0f, stddev);
                lower = __dsub_rn(mean, w);
                upper = __dadd_rn(mean, w);
            }
            const ValQD q = make_valq_d(bits, lower, upper);
            sQ = q;
            if (ONEBIT)
            {
                sLevel[0] = unquantize_d(q, bits, 0ull);
                sLevel[1] = unquantize_d(q, bits, 1ull);
            }
            double* hdr = reinterpret_cast<double*>(colp);
            hdr[0] = lower;
            hdr[1] = upper;
        }
        __syncthreads();
        // QuantizeOneQWord
        unsigned long long* __restrict__ words = reinterpret_cast<unsigned long long*>(colp + 16);
        double* ro = resOut + (long long) j * M;
        const int vpw = 64 / bits;
        const double threshold = (ONEBIT && !zeroThr) ? sQ.qmid : 0.0; // Quantize<ZeroThresholdFor1Bit> at one bit
        const double level0 = sLevel[0], level1 = sLevel[1];
        for (int t = tid; t < tasks; t += nt)
        {
            const int part = t / Q, w = t - part * Q;
            unsigned long long word = 0ull;
            unsigned i = (unsigned) t; // = w + part * Q
            for (int k = part; k < vpw && i < (unsigned) M; k += split, i += (unsigned) tasks)
            {
                const double v = resident ? sv[i] : __dadd_rn(g[i], r[i]);
                const unsigned long long qv = ONEBIT ? (v >= threshold ? 1ull : 0ull) : quantize_d(sQ, bits, v);
                ro[i] = __dsub_rn(v, ONEBIT ? (qv ? level1 : level0) : unquantize_d(sQ, bits, qv));
                word |= qv << (k * bits);
            }
            if (split == 1)
            {
                words[w] = word;
            }
            else
            {
                if ((unsigned) word)
                    atomicOr(&sWords[2 * w], (unsigned) word);
                if ((unsigned) (word >> 32))
                    atomicOr(&sWords[2 * w + 1], (unsigned) (word >> 32));
            }
        }
        if (pair)
            sv = (sv == smem) ? smem + svStride : smem; // last used two columns ago, before this column's barriers
        else if (resident || split > 1)
            __syncthreads(); // the next column may overwrite sv from here on
        if (split > 1)
            for (int w = tid; w < 2 * Q; w += nt)
            {
                reinterpret_cast<unsigned*>(words)[w] = sWords[w];
                sWords[w] = 0u;
            }
    }
}

// Shape of a quantize launch.  A CTA walks one column with two lanes, so throughput follows the columns in flight, and rows
// kept in shared memory only pay while they cost none of them.  One B200, 1 bit with threshold 0, quantize alone, us:
//                             9304 x 2048   20000 x 300   5000 x 400   512 x 363
//     1024 rows, four warps       356            286           72         10.3
//     4096 rows, eight warps      491            219           54          9.7
//     resident, eight warps       479            420           48         10.3
// (the mean threshold and the other widths order the same way).
struct ShapeD
{
    bool few;
    int threads, chunk, split, pair;
    size_t smem;
    int ctasPerSM;
};
static ShapeD launch_shape_d(long long M, long long N, int bits, int numSMs)
{
    const long long Q = (M * bits + 63) / 64;
    ShapeD s;
    auto settle = [&](bool few, int threads, long long rows, long long tasks) {
        s.few = few;
        s.threads = threads;
        s.chunk = (int) std::min(M, rows);
        s.split = (int) std::max<long long>(1, std::min<long long>(64 / bits, tasks / Q));
        s.pair = (!few && s.split == 1 && 2 * M <= rows) ? 1 : 0;
        s.smem = (size_t) ((s.chunk + 1) & ~1) * (s.pair ? 16 : 8) + (s.split > 1 ? (size_t) Q * 8 : 0);
        // 228 KB of shared memory per SM, of which a CTA also takes 1 KB for the system and the kernel's static part
        s.ctasPerSM = (int) std::min<long long>(few ? DFEW_CTAS : DMANY_CTAS * DMANY_THREADS / threads, 228 * 1024 / (long long) (s.smem + 1024 + 128));
        return N <= (long long) numSMs * s.ctasPerSM;
    };
    if (M <= DFEW_RESIDENT && settle(true, DFEW_THREADS, M, DFEW_TASKS))
        return s;
    if (settle(true, DFEW_THREADS, DFEW_CHUNK, DFEW_TASKS))
        return s;
    // two warps are enough for columns of up to 64 rows, and twice as many of them fit
    const int threads = M <= 64 ? 64 : DMANY_THREADS;
    settle(false, threads, DMANY_CHUNK, threads);
    return s;
}

// UnquantizeOneQWord (ColumnQuantizer.h:150-203), two forms.  Here: thread <-> packed word, up to 64 / bits rows of it.
__global__ void __launch_bounds__(256) k_unquantize_words_f64(const unsigned char* __restrict__ packed, double* __restrict__ out, long long M, long long N,
                                                              int bits, int add)
{
    const long long Q = (M * bits + 63) / 64;
    const long long colBytes = 16 + 8 * Q;
    const int vpw = 64 / bits;
    const long long total = N * Q;
    for (long long t = (long long) blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long) gridDim.x * blockDim.x)
    {
        const long long j = t / Q, w = t - j * Q;
        const unsigned char* colp = packed + j * colBytes;
        const ValQD q = make_valq_d(bits, reinterpret_cast<const double*>(colp)[0], reinterpret_cast<const double*>(colp)[1]);
        const unsigned long long word = reinterpret_cast<const unsigned long long*>(colp + 16)[w];
        const unsigned long long mask = q.rangeend - 1ull; // all ones when rangeend == 0 (full-word pass-through)
        double* __restrict__ o = out + j * M;
        long long i = w;
        for (int k = 0; k < vpw && i < M; ++k, i += Q)
        {
            double v = unquantize_d(q, bits, (word >> (k * bits)) & mask);
            if (add)
                v = __dadd_rn(v, o[i]);
            o[i] = v;
        }
    }
}

// Here: unit = `unitRows` consecutive rows of one column = one warp: row i is field
// i / Q of word i % Q, neighbouring lanes read neighbouring words and write neighbouring rows.  (One thread per packed word
// gives a 512 x 363 matrix 2904 threads with 64 serial, scattered stores each.)
__global__ void __launch_bounds__(256) k_unquantize_f64(const unsigned char* __restrict__ packed, double* __restrict__ out, long long M, long long N, int bits,
                                                        int add, int unitRows)
{
    const unsigned Q = (unsigned) ((M * bits + 63) / 64);
    const long long colBytes = 16 + 8 * (long long) Q;
    const long long perCol = (M + unitRows - 1) / unitRows;
    const long long total = N * perCol;
    const unsigned lane = threadIdx.x & 31;
    const unsigned advK = 32u / Q, advW = 32u - advK * Q;
    for (long long t = ((long long) blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += ((long long) gridDim.x * blockDim.x) >> 5)
    {
        const long long j = t / perCol;
        const unsigned r0 = (unsigned) (t - j * perCol) * (unsigned) unitRows;
        const unsigned end = (unsigned) min((long long) r0 + unitRows, M);
        const unsigned char* colp = packed + j * colBytes;
        const ValQD q = make_valq_d(bits, reinterpret_cast<const double*>(colp)[0], reinterpret_cast<const double*>(colp)[1]);
        const unsigned long long* __restrict__ words = reinterpret_cast<const unsigned long long*>(colp + 16);
        const unsigned long long mask = q.rangeend - 1ull; // all ones when rangeend == 0 (full-word pass-through)
        double* __restrict__ o = out + j * M;
        unsigned i = r0 + lane;
        unsigned k = i / Q, w = i - k * Q;
#pragma unroll 4
        for (; i < end; i += 32u)
        {
            double v = unquantize_d(q, bits, (words[w] >> (k * (unsigned) bits)) & mask);
            if (add)
                v = __dadd_rn(v, o[i]);
            o[i] = v;
            w += advW;
            k += advK;
            if (w >= Q)
            {
                w -= Q;
                ++k;
            }
        }
    }
}

static bool bits_ok_f64(int bits)
{
    return bits >= 1 && bits <= 64 && (bits & (bits - 1)) == 0;
}

} // namespace qagg

using namespace qagg;

extern "C" {

int64_t qagg_packed_col_bytes_f64(int64_t M, int bits)
{
    if (!bits_ok_f64(bits) || M < 0)
        return fail(QAGG_EINVAL, "qagg_packed_col_bytes_f64: bad arguments");
    return 16 + 8 * ((M * bits + 63) / 64);
}

int64_t qagg_packed_bytes_f64(int64_t M, int64_t N, int bits)
{
    if (!bits_ok_f64(bits) || M < 0 || N < 0)
        return fail(QAGG_EINVAL, "qagg_packed_bytes_f64: bad arguments");
    return N * (16 + 8 * ((M * bits + 63) / 64));
}

int qagg_quantize_f64(void* stream, const double* grad, const double* res_in, double* res_out, void* packed, int64_t M, int64_t N, int bits,
                      int zero_threshold)
{
    if (!bits_ok_f64(bits))
        return fail(QAGG_EINVAL, "bits must be a power of two in 1..64");
    if (M < 0 || N < 0 || M > 0x3fffffffLL || N > 0x7fffffffLL)
        return fail(QAGG_EINVAL, "qagg_quantize_f64: bad matrix shape");
    if (M == 0 || N == 0)
        return QAGG_OK;
    if (!grad || !res_in || !res_out || !packed)
        return fail(QAGG_EINVAL, "qagg_quantize_f64: null pointer");
    if ((reinterpret_cast<uintptr_t>(packed) & 7) || (reinterpret_cast<uintptr_t>(grad) & 7) || (reinterpret_cast<uintptr_t>(res_in) & 7) ||
        (reinterpret_cast<uintptr_t>(res_out) & 7))
        return fail(QAGG_EINVAL, "qagg_quantize_f64: buffers must be 8-byte aligned");
    LaunchCfg cfg;
    int rc = launch_cfg_for_current_device(&cfg);
    if (rc)
        return rc;
    const ShapeD sh = launch_shape_d(M, N, bits, cfg.numSMs);
    auto kern = sh.few ? (bits == 1 ? k_quantize_f64<DFEW_THREADS, DFEW_CTAS, true> : k_quantize_f64<DFEW_THREADS, DFEW_CTAS, false>)
                       : (bits == 1 ? k_quantize_f64<DMANY_THREADS, DMANY_CTAS, true> : k_quantize_f64<DMANY_THREADS, DMANY_CTAS, false>);
    if (sh.smem > 47 * 1024) // with the kernel's static part this passes the 48 KB that need no attribute
    {
        // (the same value from every thread that launches)
        rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (DFEW_RESIDENT + DFEW_TASKS) * (int) sizeof(double)),
                        "double quantize kernel attribute");
        if (rc)
            return rc;
    }
    const int grid = (int) std::min<long long>(N, (long long) cfg.numSMs * sh.ctasPerSM);
    kern<<<grid, sh.threads, sh.smem, (cudaStream_t) stream>>>(grad, res_in, res_out, static_cast<unsigned char*>(packed), (int) M, (unsigned) N, bits,
                                                               zero_threshold ? 1 : 0, sh.chunk, sh.split, sh.pair);
    return check_cuda(cudaGetLastError(), "double quantize kernel launch");
}

int qagg_unquantize_f64(void* stream, const void* packed, double* out, int64_t M, int64_t N, int bits, int add)
{
    if (!bits_ok_f64(bits))
        return fail(QAGG_EINVAL, "bits must be a power of two in 1..64");
    if (M < 0 || N < 0 || M > 0x3fffffffLL || N > 0x7fffffffLL)
        return fail(QAGG_EINVAL, "qagg_unquantize_f64: bad matrix shape");
    if (M == 0 || N == 0)
        return QAGG_OK;
    if (!packed || !out)
        return fail(QAGG_EINVAL, "qagg_unquantize_f64: null pointer");
    if ((reinterpret_cast<uintptr_t>(packed) & 7) || (reinterpret_cast<uintptr_t>(out) & 7))
        return fail(QAGG_EINVAL, "qagg_unquantize_f64: buffers must be 8-byte aligned");
    LaunchCfg cfg;
    const int rc = launch_cfg_for_current_device(&cfg);
    if (rc)
        return rc;
    // Once there are words enough for all SMs, reading each of them once is the better (us, thread per word | row units; 9304 x
    // 2048: 1 bit 31.9 | 35.6, 8 bits 33.8 | 36.7; 64 x 30000 at 8 bits 6.3 | 12.5).  Not with more bits, where a word has too few
    // rows to earn its column's range divisions (9304 x 2048: 16 bits 47.7 | 41.6, 64 bits 101 | 51.9), unless the columns are so
    // short that a row unit does not fill its warp's trips (129 x 20000 at 16 bits 8.3 | 12.4; 10 x 100000 at 64 bits 6.3 | 22.6).
    const long long words = N * ((M * bits + 63) / 64);
    if (words >= 32768 && (bits <= 8 || (bits == 16 && M <= 256) || M <= 96))
    {
        const long long grid = std::min<long long>((words + 255) / 256, (long long) cfg.numSMs * 8);
        k_unquantize_words_f64<<<(int) grid, 256, 0, (cudaStream_t) stream>>>(static_cast<const unsigned char*>(packed), out, M, N, bits, add ? 1 : 0);
        return check_cuda(cudaGetLastError(), "double unquantize kernel launch");
    }
    // 128 rows per warp while that leaves warps to spare on the chip, else 512 (fewer range divisions per value)
    const int unitRows = N * ((M + 127) / 128) <= (long long) cfg.numSMs * 64 ? 128 : 512;
    const long long total = N * ((M + unitRows - 1) / unitRows);
    const long long grid = std::min<long long>((total + 7) / 8, (long long) cfg.numSMs * 64);
    k_unquantize_f64<<<(int) grid, 256, 0, (cudaStream_t) stream>>>(static_cast<const unsigned char*>(packed), out, M, N, bits, add ? 1 : 0, unitRows);
    return check_cuda(cudaGetLastError(), "double unquantize kernel launch");
}

} // extern "C"
