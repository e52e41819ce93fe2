// Direct cross-correlation on the tensor cores (tcgen05, sm_100a), at single precision.
//
// A float is the exact sum of three bfloat16 values, x = h + m + l (8 bits of the significand each; elements from
// 2^-110 up), so a product of two floats is nine bfloat16 products, exact in the tensor cores' 32-bit accumulators.
// Six are taken.  Of the three left out, ml and lm can reach 2^-25 of the product each and ll 2^-34 (h and m are
// rounded to nearest: m is up to 2^-8 of x, l up to 2^-17); with ml and lm taken too no error measured changes.
// The accumulators round towards zero.  So the large products (hh: 16 bits, their sum of one row mostly exact) are
// summed apart from the small ones, whose rounding is 2^-8 of theirs, and both only over one right row (at most
// kTensorMaxChunk columns of it): row sums are added to nearest in registers, large and small apart, and the two sums
// meet once, when a result is written.  (All six in one accumulator: every result 0.6 to 1.2 units of 2^-24 too
// small, overlaps of up to 15 products and sparse operands off by up to twice what FFMAs lose.)  2-norm error against
// double in units of 2^-24, tile kernel -> this one: uniform operands 64 x 64 11.8 -> 2.0, 48 x 48 8.8 -> 1.7, 32 x 32
// 5.9 -> 1.4, 27 x 43 6.2 -> 1.4, one 256 x 256 pair 2.3 -> 1.5; normal 12.8 -> 2.2, 9.6 -> 1.9, 6.4 -> 1.6, 6.9 -> 1.5,
// 10.4 -> 2.7; 97 % zeros 0.57 -> 0.44, 0.51 -> 0.43, 0.46 -> 0.43, 0.46 -> 0.43, 1.15 -> 0.87; exp(4 N(0, 1)) 0.87 -> 0.79,
// 0.65 -> 0.69, 0.77 -> 0.77, 1.6 -> 1.1, 1.5 -> 1.3; and no worse at any size of the overlap (the first three kinds).
// What bias is left grows with the columns: mean error 0 for a few products, -0.4 units at 32 x 32, -0.9 at 64 x 64.
//
// As a matrix product.  One side's matrices (the "A side") are stacked to one tall matrix of rows;
// lane (row of the product) g meets row y of a matrix B of the other side with its row g + y.  Walking
// y = 0 .. H-1 a lane starts inside matrix g / H at overlap shift sy = g % H and, from y = H - sy on,
// runs on into the next matrix at shift sy - H (the last one into the first): every product of the
// cross-correlation is taken exactly once whatever H is, and a wrap costs one write of the lane's sums.
// The columns of the product are the x shifts: B's row y as a Toeplitz matrix, B[n][k] = row[x0 - n - k].
// In the unswizzled K-major layout 8 x 8 core matrices may lie anywhere, and a Toeplitz core matrix
// depends on its block row plus block column alone, so the row needs one core matrix per 8 columns
// (8 times the row's bytes, written by three producer warps from the row split once) and the two strides
// of the descriptor are the same.  A step of 16 left columns meets only W + 15 x shifts: the product's N
// is that window, and its result columns in tensor memory move with it.  What is not taken are the zeros:
// executed multiply-adds are (W + 15 rounded up to 16) / W of the definition's (1.25 at W = 64), six
// times over.  A product of N columns takes N / 2 clocks and reads (128 + N) * 32 bytes of shared memory,
// which yields 128 bytes a clock: below N = 128 the reads would set the pace.  So the columns of several
// Toeplitz matrices are interleaved in groups of 8 and taken together: of nB matrices B, or, where there
// are few, of rows y and y - 1 of the same one (nR = 2): lane g then stands for the stack's rows 2 g and
// 2 g + 1, which meet row y - rho in the same A row 2 g + y, and the A rows are staged even and odd apart.
//
// Bound by shared memory: the products alone read it at 75..95 % of its rate, and beside them a warp gets one access in
// about ten clocks; what the drain warps and the producers move comes on top.  A wrapped row costs the warp about 250
// clocks and 5 a column.  Two sums of 128 columns in two buffers fill tensor memory.  256 columns halve what the
// products read of A per result and leave room for one buffer: there the small products' sums stay in tensor memory
// from row to row and are fetched only where a lane wraps, and a row's large products, issued last, wait until those
// of the row before have been drained (48 x 48 16 x 2048 350 -> 296 us, 64 x 64 1 x 512 161 -> 152).
// Tried and left: writing a wrapped row from its lane's registers straight to global memory (one 4-byte store in
// flight per SM every 7 clocks: 64 x 64 1 x 512 took 327 us), 4 and 16 matrices interleaved (fewer wraps, but all
// warps wait for the one that writes: 32 x 32 32 x 64 88 us against 70), one sum of row totals h + small instead of two
// (sparse operands off by 0.51..0.63 units, FFMAs 0.46..0.57).
// Measured on B200 (us, tile kernel -> this one): 256 x 256 one pair 168 -> 105, 64 x 64 1 x 512 353 -> 150,
// 32 x 32 32 x 64 102 -> 82, 48 x 48 16 x 2048 449 -> 289, 27 x 43 9 x 35 54 -> 33, 256 x 256 1 x 32 4655 -> 1892.
//
// Roles of a block: the first 8 or 16 warps drain tensor memory into register sums and write results, three build the
// Toeplitz rows, the last one issues the matrix products.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cstdint>

#include "xcorr_plan.h"
#include "xcorr_launch.h"
#include "xcorr_smem.h"

namespace xcorr {

namespace {

constexpr int kProducerWarps = 3;
constexpr int kProducers = 32 * kProducerWarps;
constexpr int kRowRing = 4;                            // split rows of a B matrix kept by the producers
constexpr int kRowElems = kTensorMaxRow / kProducers;  // elements of a step's rows per producer thread
constexpr int kMaxItems = kTensorMaxItems / kProducers;  // Toeplitz rows of a step per producer thread
constexpr int kMaxSteps = kTensorMaxChunk / 16;

// Operands that are not multiplied as three bfloat16 parts, by the magnitudes of the elements a block meets:
// infinities, NaN and 2^50 upwards (products of parts must neither overflow nor meet the Toeplitz matrix's zeros as
// infinities); below 2^-110 the last part runs out of bits; and where the smallest elements of both sides have a
// product below 2^-100, products of parts can fall under the smallest normal number.  (Zeros are exact.)
constexpr unsigned kLargeBits = 0x58800000u, kTinyBits = 0x08800000u;
struct Magnitudes { unsigned large, small; };        // bits of the largest magnitude and of the smallest that is not zero
constexpr Magnitudes kNoMagnitudes = {0u, 0x7f800000u};
__device__ __forceinline__ void see(Magnitudes& m, unsigned bits) {
    bits &= 0x7fffffffu;
    m.large = max(m.large, bits);
    m.small = min(m.small, bits - 1u);               // (a zero becomes the largest number there is)
}
__device__ __forceinline__ void merge(Magnitudes* of_block, Magnitudes m) {
    m.large = __reduce_max_sync(0xffffffffu, m.large);
    m.small = __reduce_min_sync(0xffffffffu, m.small);
    if ((threadIdx.x & 31) == 0) { atomicMax(&of_block->large, m.large); atomicMin(&of_block->small, m.small); }
}
__device__ __forceinline__ bool out_of_range(const Magnitudes& a, const Magnitudes& b) {
    const unsigned least = min(a.small, b.small) + 1u;
    return max(a.large, b.large) >= kLargeBits || least < kTinyBits || ((a.small + 1u) >> 23) + ((b.small + 1u) >> 23) < 2u * 127u - 100u;
}

__device__ unsigned g_tensor_timeouts = 0;

// ---- shared memory, mbarriers, tensor memory ---------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void bar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_poll(uint32_t bar, uint32_t parity) {
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded: false after `limit` polls, or once another warp of the block has given up.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* gave_up, unsigned limit) {
    for (unsigned it = 0; it < limit; ++it) {
        if (bar_poll(bar, parity)) return true;
        if ((it & 63) == 63 && *gave_up) return false;
    }
    *gave_up = 1;
    return false;
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// KEEP: what becomes of the A operand in the tensor core's collector buffer -- read and kept for the next
// product (fill), taken from there for the last time (lastuse), or neither.
enum Keep { kDiscard, kFill, kUse, kLastUse };
#define XC_MMA(OP) \
    asm volatile("{ .reg .pred p; .reg .b64 a, b;\n\t" \
                 "mov.b64 a, {%1, %3};\n\t" \
                 "mov.b64 b, {%2, %3};\n\t" \
                 "setp.ne.b32 p, %5, 0;\n\t" \
                 "tcgen05.mma.cta_group::1.kind::f16.collector::a::" OP " [%0], a, b, %4, p; }" \
                 :: "r"(d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory")
template<Keep KEEP = kDiscard>
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
    if (KEEP == kFill) XC_MMA("fill");
    else if (KEEP == kUse) XC_MMA("use");
    else if (KEEP == kLastUse) XC_MMA("lastuse");
    else XC_MMA("discard");
}
#undef XC_MMA
// Asynchronous: the registers are the caller's after tc_load_wait.
__device__ __forceinline__ void tc_load(uint32_t addr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr));
}
// (the registers pass through it, so that nothing reads them earlier)
__device__ __forceinline__ void tc_load_wait(uint32_t (&r)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]) :: "memory");
}
__device__ __forceinline__ void tc_store(uint32_t addr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tc_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Results are written once and never read here; without a memory clobber the compiler may keep the
// shared-memory loads of the next ones in front.
__device__ __forceinline__ void put_result(float* to, float v, bool add) {
    if (add) asm volatile("red.global.add.f32 [%0], %1;" :: "l"(to), "f"(v));
    else     asm volatile("st.global.f32 [%0], %1;" :: "l"(to), "f"(v));
}
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(p));
    return p != 0;
}

// Eight floats as three vectors of eight bfloat16: v = h + m + l.
__device__ __forceinline__ void split8(const float (&v)[8], uint4 (&part)[3]) {
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = v[2 * i], b = v[2 * i + 1];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
            w[s][i] = *reinterpret_cast<const uint32_t*>(&p);
            a -= __uint_as_float(w[s][i] << 16);
            b -= __uint_as_float(w[s][i] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) part[s] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// One step of 16 columns of the A side: its product's shape, its operands and its place in tensor memory.
struct Step {
    uint32_t idesc;      // instruction descriptor with the step's N
    uint32_t b_off;      // first core matrix of the B operand, in 16-byte units from the part's start
    uint32_t d_off;      // first result column
    uint32_t a_off;      // A operand, in 16-byte units from the part's start
};

struct Shared {
    unsigned long long b_full[kTensorMaxSlots], b_empty[kTensorMaxSlots], d_full[2], d_empty[2], rest_free[2], drained;
    uint32_t tmem;
    int gave_up;
    int n_steps;
    uint32_t first_off;  // B operand of the chunk's first product, which spans all result columns
    Magnitudes a_mag, b_mag;
    Step step[kMaxSteps];
    // a drain warp's columns in the order they are written, neighbours in a result row one after the other
    // (by Toeplitz matrix, then x shift): column, and its place in its output row's image; INT_MIN: no result
    int2 column[kTensorMaxCols];
    long long row_end[2][128];                     // the output rows of a drain lane's last sums
    long long row_out[2][2][128];                  // a stack row's output rows before / after its wrap, per rho and lane; -1: none
};

// The block's place in the problem.
struct BlockTask {
    const float* a;      // the group's first A matrix
    const float* b;      // the block's first B matrix
    float* out;          // the result array, or the slice's partial image
    long long pair0;     // result matrix of (A matrix 0, the block's first B matrix)
    int row0;            // first stack row of the block
    int nb;              // B matrices of this block that exist
    int sx_lo;           // x shift of column 0
    int y0, y1;
};

// First element of the output row that stack row `srow`, matrix j of its group, belongs to before (0) or after (1) its
// wrap; -1: no such matrix.
__device__ __forceinline__ long long row_offset(const TensorPlan& p, const BlockTask& t, int srow, int j, int wrapped) {
    const int H = p.H, OW = 2 * p.W - 1, OH = 2 * H - 1;
    int g = srow / H;
    const int sy = srow - g * H - (wrapped ? H : 0);
    if (wrapped) g = (g + 1) * H < p.stack_rows ? g + 1 : 0;
    const int a = g * p.J + j, at = (sy + H - 1) * OW;
    if (srow >= p.stack_rows || a >= p.nA) return -1;
    return (t.pair0 + (long long)a * p.stride_a) * ((long long)OH * OW) + (p.flip ? OH * OW - 1 - at : at);
}

// The block's results by the definition, in single precision FMAs: operands that the split does not cover.  Only
// products that the definition has are formed (an infinity or NaN must not meet a zero that is none of the operand's).
// A warp takes 32 stack rows, one per lane, and eight x shifts of one matrix B; the A rows stand in shared memory
// as floats (as many columns at a time as fit: the results are then summed in the output), B's elements are the same
// for all lanes.  Eight elements of either side are read for 64 FMAs.  One NaN in the left matrix of 64 x 64 1 x 512
// costs 1140 us in all, where a kernel without reuse took 15.7 ms and the tile kernel takes 352 us.
__device__ __noinline__ void direct_block(const TensorArgs& args, const BlockTask t, float* smem) {
    const TensorPlan& p = args.p;
    const int H = p.H, W = p.W, OW = 2 * W - 1, OH = 2 * H - 1, J = p.J;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x >> 5;
    constexpr int kPitch = 9;                                         // of a warp's 32 x 8 results on their way out
    float* turn = smem + warp * 32 * kPitch;
    float* a_rows = smem + warps * 32 * kPitch;
    const int rows = t.y1 - t.y0, lanes = 128 * p.nR, n_staged = lanes + (rows - 1) * J;
    const int room = (int)((p.smem_bytes - (size_t)warps * 32 * kPitch * 4) / 4 / n_staged);
    const int pitch = min((room - 1) | 1, W | 1), columns = min(pitch, W);      // odd: a column of rows meets all banks
    const int row_groups = lanes / 32, units = row_groups * (p.DW / 8) * t.nb;
    for (int ua = 0; ua < W; ua += columns) {
        const int ub = min(W, ua + columns);
        __syncthreads();
        for (int i = tid; i < n_staged * (ub - ua); i += blockDim.x) {
            const int q = i / (ub - ua), u = ua + i - q * (ub - ua), sr = q / J, mat_j = q - sr * J;
            int srow = t.row0 + t.y0 + sr;
            while (srow >= p.stack_rows) srow -= p.stack_rows;
            const int g = srow / H, mat = g * J + mat_j;
            a_rows[q * pitch + u - ua] = mat < p.nA ? __ldg(t.a + ((size_t)mat * H + (srow - g * H)) * W + u) : 0.f;
        }
        __syncthreads();
        for (int unit = warp; unit < units; unit += warps) {
            const int c8 = unit / row_groups, i = (unit - c8 * row_groups) * 32 + lane, b = c8 % t.nb, sx0 = t.sx_lo + c8 / t.nb * 8;
            const int srow = t.row0 + i / J, wrap = H - srow % H;              // the row y with which this lane runs on into the next matrix
            const long long off0 = row_offset(p, t, srow, i % J, 0), off1 = row_offset(p, t, srow, i % J, 1);
            const int x_lo = max(0, ua - sx0 - 7), x_hi = min(W, ub - sx0);    // columns of B that meet the chunk at any of the shifts
            if (sx0 >= W || (x_hi <= x_lo && ua > 0)) continue;
            float acc[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = 0.f;
            // the sums of the lanes in `who` are result rows: through shared memory, so that eight neighbours leave together
            const auto put = [&](unsigned who, long long off) {
#pragma unroll
                for (int j = 0; j < 8; ++j) turn[lane * kPitch + j] = acc[j];
                __syncwarp();
                const int sx = sx0 + (lane & 7), col = p.flip ? -(sx + W - 1) : sx + W - 1;
                while (who) {
                    int src = -1;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {                              // a lane of `who` for every eight lanes
                        if (who && lane >> 3 == k) src = __ffs(who) - 1;
                        who &= who - 1;
                    }
                    const long long to = __shfl_sync(0xffffffffu, off, max(src, 0));
                    if (src >= 0 && to >= 0 && sx < W) {
                        float* o = t.out + to + b * (p.stride_b * ((long long)OH * OW)) + col;
                        const float v = turn[src * kPitch + (lane & 7)];
                        *o = ua > 0 ? *o + v : v;
                    }
                }
                __syncwarp();
            };
            const float* br = t.b + ((size_t)b * H + t.y0) * W;
            const float* ar = a_rows + i * pitch + sx0 - ua;                   // column x of B meets ar[x + j] at shift sx0 + j
            for (int y = t.y0; y < t.y1; ++y, br += W, ar += J * pitch) {
                const unsigned who = __ballot_sync(0xffffffffu, y == wrap && y > t.y0);
                if (who) {
                    put(who, off0);
                    if (y == wrap) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
                    }
                }
                float w[15];
                {
                    const int lo = ua - sx0 - x_lo, hi = ub - sx0 - x_lo;
#pragma unroll
                    for (int k = 0; k < 7; ++k) w[k + 8] = k >= lo && k < hi ? ar[x_lo + k] : 0.f;
                }
#pragma unroll 1
                for (int x = x_lo; x < x_hi; x += 8) {
                    const int lo = ua - sx0 - x, hi = ub - sx0 - x;            // elements of the window that are columns of the chunk
#pragma unroll
                    for (int k = 0; k < 7; ++k) w[k] = w[k + 8];
                    if (lo <= 0 && hi >= 15 && x + 8 <= W) {
                        float v[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) { w[k + 7] = ar[x + 7 + k]; v[k] = __ldg(br + x + k); }
#pragma unroll
                        for (int k = 0; k < 8; ++k)
#pragma unroll
                            for (int j = 0; j < 8; ++j) acc[j] = fmaf(w[k + j], v[k], acc[j]);
                    } else {
#pragma unroll
                        for (int k = 7; k < 15; ++k) w[k] = k >= lo && k < hi ? ar[x + k] : 0.f;
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            if (x + k >= W) break;
                            const float v = __ldg(br + x + k);
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                if (k + j >= lo && k + j < hi) acc[j] = fmaf(w[k + j], v, acc[j]);
                        }
                    }
                }
            }
            put(0xffffffffu, wrap < t.y1 ? off1 : off0);
        }
    }
}

// D: result columns of the block, NC for every four drain warps.  NR: rows of a B matrix taken together; with
// two, the 8-column groups belong to row offsets 0 and 1 in turn.
// MANY: the A side's columns are staged in more than one chunk (a build of its own: the sums then stay in
// registers across the whole block's code, which the single chunk's warps would pay for with spills).
template<int D, int NR, bool MANY>
__global__ void __launch_bounds__(kTensorThreads<D>, 1) tensor_kernel(const __grid_constant__ TensorArgs args) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ Shared sh;
    const TensorPlan& p = args.p;
    const int H = p.H, W = p.W, OW = 2 * W - 1, OH = 2 * H - 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kDrainWarps = kTensorDrainWarps<D>, NC = 4 * D / kDrainWarps, kMmaWarp = kDrainWarps + kProducerWarps, kThreads = kTensorThreads<D>;
    static_assert(kThreads == 32 * (kMmaWarp + 1), "block size");
    // Up to 128 columns tensor memory has two buffers for the sums of either kind, drained after every row.  256 columns
    // fill it with one: the small products' sums then stay in it, and a warp fetches them only where one of its lanes wraps.
    constexpr bool kResident = D == 256;
    constexpr uint32_t kTmemCols = kResident ? 2 * D : 4 * D;

    // ---- the block's task: x-shift tiles outermost, the heaviest (around shift 0) first
    BlockTask t;
    {
        unsigned id = blockIdx.x;
        const int slice = (int)(id % p.S); id /= p.S;
        const int bg = (int)(id % p.b_groups); id /= p.b_groups;
        const int mt = (int)(id % p.m_tiles); id /= p.m_tiles;
        const unsigned group = id % p.groups; id /= p.groups;
        const int order = (int)id, mid = (p.x_tiles - 1) / 2;
        const int xt = (order & 1) ? mid + (order + 1) / 2 : mid - order / 2;
        t.row0 = mt * (128 / p.J) * NR;
        t.nb = min(p.nB, p.nBt - bg * p.nB);
        t.sx_lo = -(W - 1) + xt * p.DW;
        t.y0 = (int)((long long)slice * H / p.S);
        t.y1 = (int)((long long)(slice + 1) * H / p.S);
        t.a = args.a + (size_t)group * p.group_a * H * W;
        t.b = args.b + ((size_t)group * p.group_b + (size_t)bg * p.nB) * H * W;
        t.pair0 = (long long)group * p.group_pairs + (long long)bg * p.nB * p.stride_b;
        t.out = args.out + (size_t)slice * args.slice_floats;
    }
    const int rows = t.y1 - t.y0;
    const int nS = p.nB * NR;                                              // Toeplitz matrices taken together
    const int steps_y = rows + NR - 1;                                   // walk of the A side
    const int n_staged = 128 / p.J * NR + rows - 1;                        // stack rows
    const int res_rows = p.res_rows;                                     // staged stack rows of one residue mod nR

    const uint32_t a_base = smem_addr(smem);
    const uint32_t a_part16 = (uint32_t)(p.KC / 8 * p.AR);                 // 16-byte units between the parts of A
    // (the final write of the results reuses the A side's space, which may have to be larger for it)
    const uint32_t b_base = a_base + max(3 * a_part16 * 16, (uint32_t)(kDrainWarps * 16 * (NC + 1) * 4));
    const int n_blk = (p.DW + p.KC) / 8;                                   // core matrices of a Toeplitz row, per B matrix
    const uint32_t b_part = (uint32_t)(n_blk * nS * 128);
    const uint32_t slot_bytes = 3 * b_part;
    const uint32_t ring_base = b_base + p.slots * slot_bytes;              // [part][row mod ring][B matrix][row_words]
    const uint32_t ring_words = (uint32_t)(kRowRing * p.nB * p.row_words);
    const int scratch_words = p.J * (NC + 4);
    float* scratch = reinterpret_cast<float*>(smem + (ring_base - a_base) + 12 * ring_words) + (warp < kDrainWarps ? warp * scratch_words : 0);

    if (tid == 0) {
        sh.gave_up = 0;
        sh.a_mag = sh.b_mag = kNoMagnitudes;
        for (int i = 0; i < p.slots; ++i) { bar_init(smem_addr(&sh.b_full[i]), kProducers); bar_init(smem_addr(&sh.b_empty[i]), 1); }
        for (int i = 0; i < 2; ++i) {
            bar_init(smem_addr(&sh.d_full[i]), 1 + args.withheld);
            bar_init(smem_addr(&sh.d_empty[i]), kDrainWarps);
            bar_init(smem_addr(&sh.rest_free[i]), kDrainWarps);
        }
        bar_init(smem_addr(&sh.drained), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // ---- result columns: 8-column groups of the nS Toeplitz matrices in turn
    for (int c = tid; c < D; c += kThreads) {
        const int blk = c >> 3, slot = blk % nS, b = slot / NR, n = blk / nS * 8 + (c & 7), sx = t.sx_lo + n;
        const int first = c / NC * (NC / 8);
        int before = 0;                            // groups of the same warp written earlier
        for (int o = first; o < first + NC / 8; ++o) before += o % nS < slot || (o % nS == slot && o < blk);
        const int at = b * (int)(p.stride_b * ((long long)OH * OW)) + (p.flip ? -(sx + W - 1) : sx + W - 1);
        sh.column[c / NC * NC + before * 8 + (c & 7)] = make_int2(c % NC, n < p.DW && b < t.nb && sx < W ? at : INT_MIN);
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&sh.tmem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;

    // ---- magnitudes of the block's B matrices (the slice's rows)
    {
        Magnitudes m = kNoMagnitudes;
        for (int b = 0; b < t.nb; ++b) {
            const unsigned* src = reinterpret_cast<const unsigned*>(t.b + ((size_t)b * H + t.y0) * W);
            for (int i = tid; i < rows * W; i += kThreads) see(m, __ldg(src + i));
        }
        merge(&sh.b_mag, m);
    }

    // ---- the lanes' output rows
    const int half_col = (warp >> 2) * NC;
    bool wrapped[NR];                              // the sums at hand belong to the shift after the wrap
    int wrap_step[NR];                             // step with which a drain lane's rows run on into the next group; -1: never
#pragma unroll
    for (int rho = 0; rho < NR; ++rho) {
        const int m = (warp & 3) * 32 + lane, srow = t.row0 + m / p.J * NR + rho, y = H - srow % H;
        wrap_step[rho] = srow < p.stack_rows && y > t.y0 && y < t.y1 ? y - t.y0 + rho : -1;
        if (warp < 4) {
            sh.row_out[0][rho][m] = row_offset(p, t, srow, m % p.J, 0);
            sh.row_out[1][rho][m] = row_offset(p, t, srow, m % p.J, 1);
        }
        wrapped[rho] = y <= t.y0;
    }

    unsigned it_base = 0;                          // rows walked before the current chunk
    int pass = 0;                                  // chunks walked
    // The chunks are walked to and fro: a stack row that does not wrap on the way keeps its sums from chunk
    // to chunk, one that does writes them at its turning point once per chunk (added from the third time on).
    // Sums of the large products and of the small ones: added to each other once, when a result is written.
    // (`rest` of the 256-column build stands in tensor memory)
    float sum[NC], rest[kResident ? 1 : NC];
    const auto no_sums = [&] {
#pragma unroll
        for (int c = 0; c < NC; ++c) { sum[c] = 0.f; if (!kResident) rest[c] = 0.f; }
    };
    if (MANY) no_sums();
    bool ok = true, covered = true;
    for (int k0 = 0; k0 < p.Kp; k0 += p.KC) {
        const int kc = min(p.KC, p.Kp - k0);
        const int X0 = p.Kp - 1 - t.sx_lo - k0;    // column of B that chunk column k meets at result column n: X0 - n - k
        // steps that meet the tile's x shifts at all; uniform over the block
        int any = 0;
        for (int s = 0; s < kc / 16; ++s) {
            const int lo = max(0, (X0 - W + 1 - 16 * s - 15) & ~7), hi = min(p.DW, X0 - 16 * s + 1);
            any |= hi > lo;
        }
        if (!any) continue;

        // ---- stage the chunk: A rows as three parts, zeros into the Toeplitz slots, the step table
        {
            // (neighbouring threads take neighbouring columns; an odd AR spreads their stores over the banks)
            const int kq = kc / 8, items = n_staged * p.J * kq;
            const uint32_t kq_rcp = (65536u + kq - 1) / kq;             // exact for the few thousand items there are
            const int first_row = t.row0 + t.y0;
            Magnitudes mag = kNoMagnitudes;
            for (int i0 = 0; i0 < items; i0 += kThreads) {
                const int i = min(i0 + tid, items - 1);                 // (the last items again rather than idle lanes)
                const int r = (int)(((uint32_t)i * kq_rcp) >> 16), q = i - r * kq;
                const int sr = r / p.J, j = r - sr * p.J;
                int srow = first_row + sr;                              // (the stack starts over behind its end)
                while (srow >= p.stack_rows) srow -= p.stack_rows;
                const int g = srow / H, mat = g * p.J + j;
                const bool there = mat < p.nA;
                const float* src = t.a + ((size_t)(there ? mat : 0) * H + (srow - g * H)) * W;
                const int u0 = p.Kp - 8 - (k0 + q * 8);                 // the item's columns: u0 + 7 down to u0
                float v[8];
                // (aligned rows in two loads: 256 x 256 pair 106.4 -> 104.7 us, 48 x 48 16 x 2048 290 -> 287, 256 x 256 1 x 32 1900 -> 1891)
                if (args.vec_ok && there && u0 + 8 <= W) {
                    const float4 lo = __ldg(reinterpret_cast<const float4*>(src + u0)), hi = __ldg(reinterpret_cast<const float4*>(src + u0 + 4));
                    v[0] = hi.w; v[1] = hi.z; v[2] = hi.y; v[3] = hi.x; v[4] = lo.w; v[5] = lo.z; v[6] = lo.y; v[7] = lo.x;
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = there && u0 + 7 - k < W ? __ldg(src + u0 + 7 - k) : 0.f;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) see(mag, __float_as_uint(v[k]));
                uint4 part[3];
                split8(v, part);
                const uint32_t at = a_base + (uint32_t)(q * p.AR + ((sr % NR) * res_rows + sr / NR) * p.J + j) * 16;
#pragma unroll
                for (int s = 0; s < 3; ++s) sts128(at + s * a_part16 * 16, part[s]);
            }
            merge(&sh.a_mag, mag);
            for (uint32_t i = tid * 16; i < p.slots * slot_bytes + 12 * ring_words; i += kThreads * 16) sts128(b_base + i, make_uint4(0, 0, 0, 0));
            if (tid == 0) {
                int n = 0;
                for (int s = 0; s < kc / 16; ++s) {
                    int lo = max(0, (X0 - W + 1 - 16 * s - 15) & ~7);
                    const int hi = min(p.DW, X0 - 16 * s + 1);
                    if (hi <= lo) continue;
                    const int cols = (hi - lo + 15) & ~15;
                    if (lo + cols > p.DW) lo = p.DW - cols;
                    Step st;
                    st.idesc = kTensorIdesc | (uint32_t)(cols * nS / 8) << 17;
                    st.b_off = (uint32_t)((2 * s + lo / 8) * nS * 8);
                    st.d_off = (uint32_t)(lo * nS);
                    st.a_off = (uint32_t)(2 * s * p.AR);
                    if (n == 0) sh.first_off = (uint32_t)(2 * s * nS * 8);
                    sh.step[n++] = st;
                }
                sh.n_steps = n;
            }
            fence_async();
            __syncthreads();
            // (what the split does not cover is not worth its products: the same for every thread)
            if (out_of_range(sh.a_mag, sh.b_mag)) { covered = false; break; }
        }

        const int back = MANY ? pass & 1 : 0;
        if (warp < kDrainWarps) {
            // ================= drain: tensor memory -> register sums -> results
            if (!MANY) no_sums();
            const uint32_t t_addr = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)half_col;
            // Stack rows that run on into the next matrices with step i: their sums so far are result rows, and the
            // next ones start from zero.
            unsigned who0 = 0, who1 = 0;
            const auto wrap_at = [&](int i) {
                const int turn = back ? steps_y - i : i;       // (backwards, the rows come back with the step before)
                who0 = __ballot_sync(0xffffffffu, turn == wrap_step[0]);
                who1 = NR == 2 ? __ballot_sync(0xffffffffu, turn == wrap_step[NR - 1]) : 0u;
                if (who0 >> lane & 1) wrapped[0] = !back;
                if (NR == 2 && (who1 >> lane & 1)) wrapped[NR - 1] = !back;
            };
            // result rows of the lanes in `now`, which stand in the warp's scratch space, written by the whole warp
            const auto write_rows = [&](unsigned now) {
                __syncwarp();
#pragma unroll
                for (int z = 0; z < NC / 32; ++z) {
                    // (with two rows taken together the first half of the order belongs to row offset 0)
                    const int2 col = sh.column[half_col + 32 * z + lane];
                    const bool second = NR == 2 && 32 * z + lane >= NC / 2;
                    for (unsigned left = now; left; left &= left - 1) {
                        const int src = __ffs(left) - 1;
                        const long long off = (second ? who1 : who0) >> src & 1 ? sh.row_out[back][second ? NR - 1 : 0][(warp & 3) * 32 + src] : -1;
                        const float v = scratch[src % p.J * (NC + 4) + col.x];
                        if (off >= 0 && col.y != INT_MIN) put_result(t.out + off + col.y, v, MANY && pass >= 2);
                    }
                }
                __syncwarp();
            };
            float4* mine = reinterpret_cast<float4*>(scratch + lane % p.J * (NC + 4));
            for (int i = 0; ok && i < steps_y; ++i) {
                const unsigned it = it_base + i;
                if (!kResident) {
                    wrap_at(i);
                    for (unsigned todo = who0 | who1; todo;) {
                        // (more than one group of J lanes where a warp's stack rows span more than H)
                        const unsigned now = todo & ((1u << p.J) - 1u) << ((__ffs(todo) - 1) & ~(p.J - 1));
                        todo &= ~now;
                        if (now >> lane & 1) {
#pragma unroll
                            for (int c = 0; c < NC; c += 4)
                                mine[c / 4] = make_float4(sum[c] + rest[kResident ? 0 : c], sum[c + 1] + rest[kResident ? 0 : c + 1],
                                                          sum[c + 2] + rest[kResident ? 0 : c + 2], sum[c + 3] + rest[kResident ? 0 : c + 3]);
                        }
                        write_rows(now);
                    }
                }
                const int buffer = kResident ? 0 : it & 1;
                if (kResident) {
                    // The next row's small products may be added to the sums that stay in tensor memory (rest_free) once the
                    // lanes that wrap with it have taken theirs: at once where there are none.  Two barriers in turn: a warp
                    // can be a row ahead of the products here, not two (d_full of this row comes before the row after next).
                    if (i + 1 < steps_y) wrap_at(i + 1); else who0 = who1 = 0;
                    if (!(who0 | who1) && lane == 0) bar_arrive(smem_addr(&sh.rest_free[it & 1]));
                }
                ok = bar_wait(smem_addr(&sh.d_full[buffer]), (kResident ? it : it >> 1) & 1, &sh.gave_up, args.wait_limit);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                if (kResident) {
#pragma unroll
                    for (int c0 = 0; c0 < NC; c0 += 16) {
                        uint32_t v[8], w[8];
                        tc_load(t_addr + c0, v);
                        tc_load(t_addr + c0 + 8, w);
                        tc_load_wait(v);
                        tc_load_wait(w);
#pragma unroll
                        for (int c = 0; c < 8; ++c) { sum[c0 + c] += __uint_as_float(v[c]); sum[c0 + 8 + c] += __uint_as_float(w[c]); }
                    }
                    // Lanes that wrap with the next row (one group of J at most, by the plan).  No products run until this is
                    // done: beside them a warp gets one access to shared memory in about ten clocks.
                    if (who0 | who1) {
#pragma unroll
                        for (int c0 = 0; c0 < NC; c0 += 8) {
                            const unsigned who = NR == 2 && (c0 & 8) ? who1 : who0;      // (eight columns belong to one row offset)
                            if (!who) continue;
                            uint32_t w[8];
                            tc_load(t_addr + D + c0, w);
                            tc_load_wait(w);
                            if (who >> lane & 1) {
                                float f[8];
#pragma unroll
                                for (int c = 0; c < 8; ++c) { f[c] = sum[c0 + c] + __uint_as_float(w[c]); sum[c0 + c] = 0.f; w[c] = 0u; }
                                mine[c0 / 4] = make_float4(f[0], f[1], f[2], f[3]);
                                mine[c0 / 4 + 1] = make_float4(f[4], f[5], f[6], f[7]);
                            }
                            tc_store(t_addr + D + c0, w);
                        }
                        tc_store_wait();
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (who0 | who1) bar_arrive(smem_addr(&sh.rest_free[it & 1]));
                        bar_arrive(smem_addr(&sh.d_empty[0]));
                    }
                    if (who0 | who1) write_rows(who0 | who1);
                } else {
                    const float keep0 = who0 >> lane & 1 ? 0.f : 1.f, keep1 = who1 >> lane & 1 ? 0.f : 1.f;
#pragma unroll
                    for (int c0 = 0; c0 < NC; c0 += 8) {
                        uint32_t v[8], w[8];
                        tc_load(t_addr + buffer * 2 * D + c0, v);
                        tc_load(t_addr + buffer * 2 * D + D + c0, w);
                        tc_load_wait(v);
                        tc_load_wait(w);
                        // (eight columns belong to one row offset; exact: times 1 or 0)
                        const float keep = NR == 2 && (c0 & 8) ? keep1 : keep0;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            sum[c0 + c] = fmaf(sum[c0 + c], keep, __uint_as_float(v[c]));
                            rest[kResident ? 0 : c0 + c] = fmaf(rest[kResident ? 0 : c0 + c], keep, __uint_as_float(w[c]));
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(smem_addr(&sh.d_empty[buffer]));
                }
            }
        } else if (warp < kMmaWarp) {
            // ================= producers: row y of every B matrix of the block as a Toeplitz matrix
            // A row is split once and kept reversed as three runs of bfloat16 (element e is column X0 - e);
            // row n of core matrix i is the eight elements from e = 8 i + n on.
            const int ptid = tid - 32 * kDrainWarps;
            const int i_lo = max(0, (X0 - W + 1 - 14 + 7) >> 3), i_hi = min(n_blk - 1, X0 >> 3);
            const int items = max(0, i_hi - i_lo + 1) * nS * 8, row_elems = t.nb * W;
            const int e_end = 8 * (i_hi - i_lo + 1) + 8;
            const uint32_t part_bytes = 4 * ring_words, row_bytes = (uint32_t)p.row_words * 4;
            float ahead[kRowElems];
            uint32_t at[kRowElems];               // byte offset of the element in a ring row set; ~0: not needed
            const float* from[kRowElems];
#pragma unroll
            for (int j = 0; j < kRowElems; ++j) {
                const int idx = ptid + j * kProducers, b = idx / W, x = idx - b * W;
                const int e = X0 - x - 8 * i_lo;
                at[j] = idx < row_elems && e >= 0 && e < e_end ? (uint32_t)b * row_bytes + 2u * (uint32_t)e : ~0u;
                from[j] = t.b + ((size_t)b * H + t.y0) * W + x;
                if (back) from[j] += (size_t)(rows - 1) * W;
                ahead[j] = at[j] != ~0u ? __ldg(from[j]) : 0.f;
            }
            // the thread's Toeplitz rows: where they are read in a ring row and written in a slot
            uint32_t item[kMaxItems], item_dst[kMaxItems];
#pragma unroll
            for (int j = 0; j < kMaxItems; ++j) {
                const int e = ptid + j * kProducers, n = e & 7, blk = e >> 3, bi = blk / nS, sl = blk - bi * nS, b = sl / NR;
                item[j] = (uint32_t)b * row_bytes + (uint32_t)(4 * bi + (n >> 1)) * 4 + (NR == 2 ? (uint32_t)(sl & 1) << 31 : 0u);
                item_dst[j] = (uint32_t)((i_lo * nS + blk) * 128 + n * 16);
            }
            const uint32_t shift = (ptid & 1) * 16;
            // (a warp that gave up a wait keeps meeting the others at the barrier)
            for (int i = 0; i < steps_y; ++i) {
                const unsigned it = it_base + i, use = it / p.slots;
                const int slot = (int)(it - use * p.slots);
                // step's place in the walk, and the row it brings: the first of its rows, or backwards the last
                const int place = back ? steps_y - 1 - i : i, fresh = back ? place - (NR - 1) : place;
                const uint32_t ring_row = ring_base + (uint32_t)(fresh & (kRowRing - 1)) * (uint32_t)p.nB * row_bytes;
                const bool real = fresh >= 0 && fresh < rows;
#pragma unroll
                for (int j = 0; j < kRowElems; ++j) {
                    if (at[j] == ~0u) continue;
                    float v = real ? ahead[j] : 0.f;              // (beyond the first and last row: zeros)
#pragma unroll
                    for (int s = 0; s < 3; ++s) {
                        const __nv_bfloat16 h = __float2bfloat16_rn(v);
                        asm volatile("st.shared.b16 [%0], %1;" :: "r"(ring_row + at[j] + s * part_bytes),
                                     "h"(__bfloat16_as_ushort(h)) : "memory");
                        v -= __bfloat162float(h);
                    }
                    if (i + 1 < rows) ahead[j] = __ldg(from[j] + (back ? -(long long)(i + 1) * W : (long long)(i + 1) * W));
                }
                asm volatile("bar.sync 1, %0;" :: "n"(kProducers) : "memory");
                if (ok && use > 0) ok = bar_wait(smem_addr(&sh.b_empty[slot]), (use - 1) & 1, &sh.gave_up, args.wait_limit);
                ok = __all_sync(0xffffffffu, ok);
                const uint32_t dst0 = b_base + slot * slot_bytes, set_bytes = (uint32_t)p.nB * row_bytes;
                const uint32_t src0 = ring_base + (uint32_t)(place & (kRowRing - 1)) * set_bytes;
                const uint32_t src1 = ring_base + (uint32_t)((place - 1) & (kRowRing - 1)) * set_bytes;
                if (ok) {
#pragma unroll
                    for (int j = 0; j < kMaxItems; ++j) {
                        if (j * kProducers >= items) break;
                        if (ptid + j * kProducers >= items) continue;
                        const uint32_t src = NR == 2 ? ((int)item[j] < 0 ? src1 : src0) + (item[j] & 0x7fffffffu) : src0 + item[j];
                        uint32_t w[3][5];
#pragma unroll
                        for (int s = 0; s < 3; ++s)
#pragma unroll
                            for (int k = 0; k < 5; ++k)
                                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[s][k]) : "r"(src + s * part_bytes + 4 * k));
#pragma unroll
                        for (int s = 0; s < 3; ++s)
                            sts128(dst0 + item_dst[j] + s * b_part,
                                   make_uint4(__funnelshift_r(w[s][0], w[s][1], shift), __funnelshift_r(w[s][1], w[s][2], shift),
                                              __funnelshift_r(w[s][2], w[s][3], shift), __funnelshift_r(w[s][3], w[s][4], shift)));
                    }
                }
                fence_async();
                bar_arrive(smem_addr(&sh.b_full[slot]));
            }
            if (MANY) no_sums();                      // (the other roles keep no registers for them)
        } else {
            // ================= matrix products: one row of B against 128 rows of A
            const bool leader = elect_one();
            const uint32_t desc_hi = 8u | 1u << 14;                       // 128 bytes between groups of 8 rows; descriptor version
            const uint32_t a_lo0 = (a_base >> 4) | (uint32_t)p.AR << 16, lbo_b = (uint32_t)(8 * nS) << 16;
            const uint32_t idesc_all = kTensorIdesc | (uint32_t)(p.DW * nS / 8) << 17;
            const uint32_t bp = b_part >> 4, first_off = sh.first_off;
            const int n_steps = sh.n_steps;
            Step st[kMaxSteps];
#pragma unroll
            for (int s = 0; s < kMaxSteps; ++s) st[s] = sh.step[s < n_steps ? s : 0];
            for (int i = 0; ok && i < steps_y; ++i) {
                const unsigned it = it_base + i, use = it / p.slots;
                const int slot = (int)(it - use * p.slots);
                ok = bar_wait(smem_addr(&sh.b_full[slot]), use & 1, &sh.gave_up, args.wait_limit);
                if (kResident && ok && it >= 1) ok = bar_wait(smem_addr(&sh.rest_free[(it - 1) & 1]), ((it - 1) >> 1) & 1, &sh.gave_up, args.wait_limit);
                if (!kResident && ok && it >= 2) ok = bar_wait(smem_addr(&sh.d_empty[it & 1]), ((it >> 1) - 1) & 1, &sh.gave_up, args.wait_limit);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const int place = back ? steps_y - 1 - i : i;
                const uint32_t a0 = a_lo0 + ((place % NR) * res_rows + place / NR) * p.J;
                const uint32_t large = tmem + (kResident ? 0 : it & 1) * 2 * D, small = large + D;
                const uint32_t b0 = ((b_base + slot * slot_bytes) >> 4) | lbo_b;
                // The first product of a row into either sum spans all result columns (against the Toeplitz matrix's
                // zeros outside its window) and overwrites the buffer; the sums that stay there start with the first row.
                if (leader) {
                    tc_mma(small, a0 + st[0].a_off + 2 * a_part16, b0 + first_off, desc_hi, idesc_all, kResident && it > 0);
#pragma unroll
                    for (int s = 0; s < kMaxSteps; ++s) {
                        if (s >= n_steps) break;
                        const uint32_t a = a0 + st[s].a_off, b = b0 + st[s].b_off, d = small + st[s].d_off, id = st[s].idesc;
                        if (s > 0) tc_mma(d, a + 2 * a_part16, b, desc_hi, id, 1);
                        // (the middle and the high part of A are each read once for two products or three)
                        tc_mma<kFill>(d, a + a_part16, b + bp, desc_hi, id, 1);
                        tc_mma<kLastUse>(d, a + a_part16, b, desc_hi, id, 1);
                        tc_mma<kFill>(d, a, b + 2 * bp, desc_hi, id, 1);
                        if (kResident || s == 0) {
                            tc_mma<kLastUse>(d, a, b + bp, desc_hi, id, 1);
                        } else {
                            tc_mma<kUse>(d, a, b + bp, desc_hi, id, 1);
                            tc_mma<kLastUse>(large + st[s].d_off, a, b, desc_hi, id, 1);
                        }
                        if (!kResident && s == 0) tc_mma(large, a, b0 + first_off, desc_hi, idesc_all, 0);
                    }
                }
                __syncwarp();
                if (kResident) {
                    // the large products last: their sums of the row before are drained meanwhile
                    if (it >= 1) ok = bar_wait(smem_addr(&sh.d_empty[0]), (it - 1) & 1, &sh.gave_up, args.wait_limit);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) {
                        tc_mma(large, a0 + st[0].a_off, b0 + first_off, desc_hi, idesc_all, 0);
#pragma unroll
                        for (int s = 1; s < kMaxSteps; ++s) {
                            if (s >= n_steps) break;
                            tc_mma(large + st[s].d_off, a0 + st[s].a_off, b0 + st[s].b_off, desc_hi, st[s].idesc, 1);
                        }
                    }
                }
                if (leader) {
                    tc_commit(smem_addr(&sh.b_empty[slot]));
                    tc_commit(smem_addr(&sh.d_full[kResident ? 0 : it & 1]));
                }
                __syncwarp();
            }
            if (MANY) no_sums();
        }
        it_base += steps_y;
        ++pass;
        tc_fence_before();
        if (__syncthreads_or(!ok)) { ok = false; break; }
        tc_fence_after();
        if (!MANY) break;
    }

    // ---- the walk's end: all sums are result rows.  Through shared memory (the A side is done with: all
    // products have completed), 16 lanes at a time, so that a store instruction writes up to 32 neighbours.
    if (ok && covered && warp < kDrainWarps) {
        float* tile = reinterpret_cast<float*>(smem) + warp * 16 * (NC + 1);
        if (kResident) {
            const uint32_t t_addr = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)half_col + D;
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += 8) {
                uint32_t w[8];
                tc_load(t_addr + c0, w);
                tc_load_wait(w);
#pragma unroll
                for (int c = 0; c < 8; ++c) sum[c0 + c] += __uint_as_float(w[c]);
            }
            tc_fence_before();
        }
        // (the warps of the same lanes set the same values)
        unsigned again[NR];                        // rows that wrapped on the way have been written before, unless this was the only pass
#pragma unroll
        for (int rho = 0; rho < NR; ++rho) {
            again[rho] = MANY && pass > 1 ? __ballot_sync(0xffffffffu, wrap_step[rho] >= 0) : 0u;
            sh.row_end[rho][(warp & 3) * 32 + lane] = sh.row_out[wrapped[rho] ? 1 : 0][rho][(warp & 3) * 32 + lane];
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            if (lane >> 4 == half) {
#pragma unroll
                for (int c = 0; c < NC; ++c) tile[(lane & 15) * (NC + 1) + c] = kResident ? sum[c] : sum[c] + rest[kResident ? 0 : c];
            }
            __syncwarp();
#pragma unroll 1
            for (int z = 0; z < NC / 32; ++z) {
                const int2 col = sh.column[half_col + 32 * z + lane];
                if (col.y != INT_MIN) {
                    const bool second = NR == 2 && 32 * z + lane >= NC / 2;
                    const long long* offs = &sh.row_end[second ? 1 : 0][(warp & 3) * 32 + half * 16];
                    const unsigned ag = MANY ? again[second ? NR - 1 : 0] >> (half * 16) : 0u;
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const long long off = offs[r];
                        const float v = tile[r * (NC + 1) + col.x];
                        if (off >= 0) put_result(t.out + off + col.y, v, ag >> r & 1);
                    }
                }
            }
            __syncwarp();
        }
    }

    // ---- operands the split does not cover: the block's results again, by the definition
    __syncthreads();
    if (warp == kMmaWarp) {
        if (!ok) {
            // products may be in flight: let them land before their memory goes (with the full limit, whatever the others had)
            if (elect_one()) tc_commit(smem_addr(&sh.drained));
            __syncwarp();
            for (unsigned it = 0; it < kStageWaitLimit && !bar_poll(smem_addr(&sh.drained), 0); ++it) {}
            __syncwarp();
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTmemCols) : "memory");
    }
    if (!ok) {
        if (tid == 0) atomicAdd(&g_tensor_timeouts, 1u);
        return;
    }
    if (!covered) {
        direct_block(args, t, reinterpret_cast<float*>(smem));
        return;
    }
    // ---- the corners of a result are single products: rounded once, as the definition has them (the three
    // products of parts left out and the rounding towards zero would show in their last bit)
    for (int i = tid; i < 128 * NR * t.nb * 2; i += kThreads) {
        const int right_side = i & 1, b = (i >> 1) % t.nb, m = (i >> 1) / t.nb;
        const int srow = t.row0 + m / p.J, cy = srow % H, sx = right_side ? W - 1 : 1 - W;
        if (srow >= p.stack_rows || sx < t.sx_lo || sx >= t.sx_lo + p.DW) continue;
        int g = srow / H;
        const bool bottom = cy == H - 1 && t.y0 == 0, top = cy == 1 && t.y1 == H;       // shift H - 1 / 1 - H
        if (!bottom && !top) continue;
        if (top) g = (g + 1) * H < p.stack_rows ? g + 1 : 0;
        const int a = g * p.J + m % p.J;
        if (a >= p.nA) continue;
        const float av = __ldg(t.a + ((size_t)a * H + (bottom ? H - 1 : 0)) * W + (right_side ? W - 1 : 0));
        const float bv = __ldg(t.b + ((size_t)b * H + (bottom ? 0 : H - 1)) * W + (right_side ? 0 : W - 1));
        const int at = (bottom ? OH - 1 : 0) * OW + (right_side ? OW - 1 : 0);
        const long long pair = t.pair0 + (long long)a * p.stride_a + (long long)b * p.stride_b;
        t.out[pair * ((long long)OH * OW) + (p.flip ? OH * OW - 1 - at : at)] = av * bv;
    }
}

int up(int v, int m) { return (v + m - 1) / m * m; }

}  // namespace

cudaError_t launch_tensor(const TensorArgs& a, int device, cudaStream_t stream) {
    void (*const kernels[2][2][3])(TensorArgs) = {
        {{tensor_kernel<64, 1, false>, tensor_kernel<128, 1, false>, tensor_kernel<256, 1, false>},
         {tensor_kernel<64, 1, true>, tensor_kernel<128, 1, true>, tensor_kernel<256, 1, true>}},
        {{tensor_kernel<64, 2, false>, tensor_kernel<128, 2, false>, tensor_kernel<256, 2, false>},
         {tensor_kernel<64, 2, true>, tensor_kernel<128, 2, true>, tensor_kernel<256, 2, true>}}};
    const int many = a.p.Kp > a.p.KC ? 1 : 0, cols = a.p.D / 128;
    auto* kernel = kernels[a.p.nR - 1][many][cols];
    static SmemLimit limits[2][2][3];
    const cudaError_t e = limits[a.p.nR - 1][many][cols].allow(device, a.p.smem_bytes, [&](size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
    if (e != cudaSuccess) return e;
    kernel<<<a.p.grid, tensor_threads(a.p.D), a.p.smem_bytes, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t tensor_wait_timeouts(unsigned* count) {
    unsigned zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(count, g_tensor_timeouts, sizeof *count);
    if (e == cudaSuccess && *count != 0) e = cudaMemcpyToSymbol(g_tensor_timeouts, &zero, sizeof zero);
    return e;
}

bool plan_tensor(const PairMap& pm, int H, int W, int sm_count, int max_slices, double max_err2, TensorPlan* out, double* out_us) {
    if (H < 8 || W < 8 || H > 1024 || W > kTensorMaxRow) return false;
    const bool shared_rights = pm.n_left == 1 || pm.right_stride == 0;     // every left meets every right
    double best = 1e30;
    for (int flip = 0; flip < 2; ++flip) {
        TensorPlan p{};
        p.H = H; p.W = W; p.flip = flip;
        const unsigned m = pm.m, n = pm.n_left;
        if (shared_rights) {
            p.groups = 1;
            p.nA = (int)(flip ? m : n); p.nBt = (int)(flip ? n : m);
            p.stride_a = (int)(flip ? 1 : m); p.stride_b = (int)(flip ? m : 1);
        } else {
            p.groups = n;
            p.nA = (int)(flip ? m : 1); p.nBt = (int)(flip ? 1 : m);
            p.stride_a = flip ? 1 : 0; p.stride_b = flip ? 0 : 1;
            p.group_a = (int)(flip ? m : 1); p.group_b = (int)(flip ? 1 : m); p.group_pairs = (int)m;
        }
        if ((long long)p.nA * H > 1 << 30) continue;
        p.Kp = up(W, 16);
        for (int D = 64; D <= kTensorMaxCols; D *= 2)
        for (int nB = 1; nB <= std::min(p.nBt, kTensorMaxB); ++nB)
        for (int nR = 1; nR <= (nB == 1 ? 2 : 1); ++nR)
        for (int J = 1; J <= std::min(p.nA, kTensorMaxJ); J *= 2)
        for (int S = 1; S <= std::min(max_slices, H); ++S) {
            if (S > 1 && (flip || p.nA != 1)) break;
            if (nB * W > kTensorMaxRow) continue;
            const int nS = nB * nR;
            const int dw = D / nS / 16 * 16;
            if (dw < 16) break;
            p.D = D; p.nB = nB; p.nR = nR; p.S = S; p.J = J;
            p.stack_rows = (p.nA + J - 1) / J * H;
            p.m_tiles = (unsigned)((p.stack_rows + 128 / J * nR - 1) / (128 / J * nR));
            p.x_tiles = (2 * W - 1 + dw - 1) / dw;
            p.DW = up((2 * W - 1 + p.x_tiles - 1) / p.x_tiles, 16);
            p.b_groups = (unsigned)((p.nBt + nB - 1) / nB);
            const int rows = (H + S - 1) / S;
            // a split row: W elements, what the last core matrix reads beyond them, zeros
            p.row_words = up((W + 14) / 8 * 8 + 8 + 16, 8) / 2;
            p.res_rows = (128 / J * nR + rows - 1 + nR - 1) / nR;
            p.AR = nR * p.res_rows * J | 1;
            // Toeplitz rows of a step, whatever the tile
            if (((W + 13) / 8 + 1) * nS * 8 > kTensorMaxItems) continue;
            const int drain_warps = tensor_threads(D) / 32 - 4, NC = 4 * D / drain_warps;
            // (256 columns: one group of J lanes of a warp at most wraps at a time -- groups g and g' do together where
            // nR * (g - g') is a multiple of H)
            if (D == 256 && 32 / J > H / (H % nR == 0 ? nR : 1)) continue;
            const auto smem_of = [&] {
                const size_t a_bytes = std::max<size_t>((size_t)3 * (p.KC / 8) * p.AR * 16, (size_t)drain_warps * 16 * (NC + 1) * 4);
                return a_bytes + (size_t)p.slots * 3 * ((p.DW + p.KC) / 8) * nS * 128 + (size_t)drain_warps * J * (NC + 4) * 4 +
                       (size_t)12 * kRowRing * nB * p.row_words;
            };
            bool fits = false;
            for (p.slots = kTensorMaxSlots; p.slots >= 2; --p.slots) {
                for (p.KC = std::min(p.Kp, kTensorMaxChunk); p.KC >= (p.slots > 2 ? std::min(p.Kp, 48) : 16); p.KC -= 16)
                    if (smem_of() <= kSmemLimit - sizeof(Shared) - 1024) { fits = true; break; }
                if (fits) break;
            }
            if (!fits) continue;
            const int chunks = (p.Kp + p.KC - 1) / p.KC;
            p.KC = up((p.Kp + chunks - 1) / chunks, 16);
            // (two rows together in 256 columns over several chunks: never within 5 % of the best plan timed)
            if (D == 256 && nR == 2 && chunks > 1) continue;
            // the sums in registers, one per row and chunk, taken one after the other in every slice (64 x 64: 1.97 measured,
            // 2.05 by this; 256 x 256 in 37 slices 1.72, 1.61); rounding once and what the products leave out
            const double sums = (double)H * chunks;
            if (0.3 + 0.061 * (sums / ((double)S * S) + S) > max_err2) continue;
            // one block per SM: half of tensor memory or more, and the registers, are taken
            p.smem_bytes = std::max<size_t>(smem_of(), 120 * 1024);
            if ((double)nB * p.stride_b * (2.0 * H - 1) * (2.0 * W - 1) > 2e9) continue;    // (32-bit column offsets)
            const unsigned long long grid = (unsigned long long)p.x_tiles * p.groups * p.m_tiles * p.b_groups * S;
            if (grid > 0x7fffffffull) continue;
            p.grid = (unsigned)grid;
            // Time of a block in clocks: its matrix products at the tensor cores' rate or that of the shared memory they
            // read, its Toeplitz rows, its drains and wrapped rows; of these the longest, and most of the second, since
            // all of them share the memory.  Constants fitted to 2313 plans timed on 90 shapes (4 % in the mean square).
            const double together = H % nR == 0 ? nR : 1;       // every so many steps several lanes of a block wrap at once
            const double some = std::min(1.0 / together, 128.0 / J / H);                  // steps in which any does
            const double wraps = some * std::max(1.0, 32.0 / J / H * together);           // groups of a warp, one after the other
            const double wrap_clk = 248.0 + 5.3 * NC;
            double sum_clk = 0, max_clk = 0, tile_clk[64];
            const int xt_n = std::min(p.x_tiles, 64);
            for (int xt = 0; xt < xt_n; ++xt) {
                double clk = 100.0 + 130.0 * D;
                for (int k0 = 0; k0 < p.Kp; k0 += p.KC) {
                    const int kc = std::min(p.KC, p.Kp - k0);
                    const int X0 = p.Kp - 1 + W - 1 - xt * p.DW - k0;
                    double row = 0;
                    for (int s = 0; s < kc / 16; ++s) {
                        const int lo = std::max(0, (X0 - W + 1 - 16 * s - 15) & ~7), hi = std::min(p.DW, X0 - 16 * s + 1);
                        if (hi <= lo) continue;
                        const double cols = (double)up(hi - lo, 16) * nS;
                        row += 6 * std::max(cols / 2, (D == 256 ? 21 : 16) + cols / 4) + (row == 0 ? p.DW * nS - cols : 0);
                    }
                    if (row == 0) continue;
                    const int blocks = std::min((W + 13) / 8 + 1, (p.DW + kc) / 8);
                    double produce = 233.0 + 225.0 * ((blocks * nS * 8 + kProducers - 1) / kProducers) + 120.0 * ((nB * W + kProducers - 1) / kProducers);
                    if (p.Kp > p.KC && D >= 128) produce += D == 128 ? 670.0 : 1540.0;    // (these builds spill)
                    double drain = 6.4 * D;
                    if (D == 256) {
                        row = 0.95 * row + 15.0 + some * 830.0;
                        drain += 0.57 * wraps * J * wrap_clk;
                    } else {
                        row = 0.95 * row + 40.0;
                        drain += wraps * (1.0 + 0.16 * (J - 1)) * wrap_clk;
                    }
                    double c3[3] = {row, produce, drain};
                    std::sort(c3, c3 + 3);
                    clk += (rows + nR - 1) * (c3[2] + 0.66 * c3[1]) + 4.3 * p.AR * (kc / 8) + 6500.0;
                }
                tile_clk[xt] = clk;
                sum_clk += clk;
                max_clk = std::max(max_clk, clk);
            }
            const double total = sum_clk * ((double)p.grid / xt_n);
            const double waves = (double)p.grid / sm_count;
            double us = 4.7;
            if (S > 1) us += 2.0 + (double)S * (2.0 * H - 1) * (2.0 * W - 1) * p.nBt * 4 / 4e6;
            if (us + std::max(max_clk, total / sm_count) / 1850.0 >= best) continue;
            // the busiest SM: whole blocks, each to the SM that is free first, in the order of the launch (a tile's blocks are alike)
            double clk = total / sm_count + 0.2 * max_clk;
            if (waves <= 12 && p.x_tiles <= 64 && sm_count <= 256) {
                double load[256] = {};
                const int per_tile = (int)(p.grid / (unsigned)p.x_tiles), mid = (p.x_tiles - 1) / 2;
                for (int o = 0; o < p.x_tiles; ++o) {
                    const double c = tile_clk[(o & 1) ? mid + (o + 1) / 2 : mid - o / 2];
                    for (int i = 0; i < sm_count; ++i) load[i] += c * (per_tile / sm_count + (i < per_tile % sm_count ? 1 : 0));
                    if (per_tile % sm_count) std::sort(load, load + sm_count);
                }
                clk = *std::max_element(load, load + sm_count);
            }
            us += clk / 1850.0;
            if (us < best) { best = us; *out = p; }
        }
    }
    *out_us = best;
    return best < 1e29;
}

}  // namespace xcorr
