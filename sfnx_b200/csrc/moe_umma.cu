// The routed experts over many rows (the prompt path's jobs of up to 64 rows of one expert) on Blackwell's fifth-generation
// tensor cores.  Replaces reference src/moe_mma.cu:28-59 / src/moe_mma.cuh:63-379 (moe_gate_up_mma, swiglu_h16,
// moe_down_mma; HMMA.884 there).
//
// The values are the reference's: each weight dequantised to f16 with one rounding (Q4_K: the sub-block scale d sc and
// min dmin m rounded to f16, then one half fma q * f16(d sc) - f16(dmin m), src/moe_mma.cuh:56-60, 79-113; Q8_0: one
// half product q * d, :184-216; Q6_K in 32-column units, which the reference's prompt path does not take, by the same
// rule: one half product (q - 32) * f16(d sc)), activations f16, products summed in fp32.
//
// One persistent CTA a multiprocessor walks tiles of 256 of an expert's rows against one or two of the expert's jobs
// (consecutive jobs of one expert are paired, so that their weights are dequantised once), the tiles of a pair side by side
// on neighbouring CTAs.  The rows are the M side of tcgen05.mma (kind::f16, cta_group::1, twice M 128), the jobs'
// activation rows the N side (16 to 128), and the 256 x N fp32 result sits in one of two halves of tensor memory.
//   warps 0-15   the producers: 64 columns at a time of the weights into the A operand (rows of 128 bytes, K-major, 128-byte
//                swizzle) in one of three shared-memory stages.  A tile's result is written out after the next
//                tile's first stages are full, so the tensor cores and the copies never wait for it.
//   warp 16      issues a full stage's MMAs (K 16 each) and lets tcgen05.commit hand the stage back
//   warp 17      copies the raw weights (asynchronous copies into a ring of their own)
//   warps 18-23  the jobs' activation rows (the B operand, same form) by asynchronous copies, two warps a stage
// Every wait is bounded and feeds the device fault word.
//
// What bounds it: the producers' dequantisation and the shared-memory pipe (its stores and the weights' 16-byte loads), not
// the tensor cores or HBM.  256 rows a tile halve the copies of activation rows (against 128 rows and two CTAs an SM), and
// running on from tile to tile hides a tile's start and end.  4096 tokens (1010 jobs, 512 experts
// of 1536 x 3072 and 3072 x 768): gate|up Q4_K 1.18 -> 0.84 ms, down Q6_K 0.95 -> 0.64; Q8_0 1.42 -> 0.89 and 0.92 -> 0.50;
// 130 tokens, Q4_K/Q6_K: 0.92 -> 0.54 and 0.64 -> 0.48.
#include <algorithm>

#include "common.cuh"
#include "copy_ring.h"
#include "exact_math.cuh"
#include "moe_internal.cuh"
#include "umma.cuh"

namespace fnxk {

constexpr int MU_BM = 256, MU_KC = 64, MU_NS = 3, MU_PROD = 512, MU_COPY = 6, MU_THREADS = MU_PROD + 64 + 32 * MU_COPY, MU_PAIR = 2, MU_NMAX = MU_PAIR * FNX_PF_JOB;
constexpr int MU_LIST = 2048;   // jobs whose pairs are listed at a time
constexpr int MU_ABYTES = MU_BM * 128, MU_BBYTES = MU_NMAX * 128, MU_STAGE = MU_ABYTES + MU_BBYTES;
constexpr int MU_RAW = 73728;   // the raw weights' ring
constexpr size_t MU_SMEM = (size_t) MU_NS * MU_STAGE + MU_RAW + 1024 + MU_LIST * 2;

__device__ __forceinline__ void mu_arrive(unsigned long long* bar) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(um_s32(bar)) : "memory");
}

// four bytes (each 0..255) as f16 pairs {b0, b1}, {b2, b3} less `bias`: 0x6400 | b is the f16 1024 + b exactly
__device__ __forceinline__ void mu_bytes(unsigned w, __half2 bias, __half2& lo, __half2& hi) {
    const unsigned p = __byte_perm(w, 0x64646464u, 0x4140), q = __byte_perm(w, 0x64646464u, 0x4342);
    lo = __hsub2(*reinterpret_cast<const __half2*>(&p), bias);
    hi = __hsub2(*reinterpret_cast<const __half2*>(&q), bias);
}
__device__ __forceinline__ __half2 mu_h2(unsigned short bits) { return __half2half2(__ushort_as_half(bits)); }
__device__ __forceinline__ unsigned mu_u(__half2 h) { return *reinterpret_cast<const unsigned*>(&h); }

struct MuArgs {
    int type, nrows, ncols;
    const unsigned char *a, *b, *c, *d;
    size_t stride, stride_b;
    const FnxBigJob* jobs;
    const int* njobs;
    int njobs_cap;   // jobs past it are the caller's other memory, whatever the count on the device says
    const uint16_t* x;
    float* out;
    unsigned* fault;
};

// The raw weights of a tile: the plane that holds nearly all of them comes through a ring in shared memory, STEPS steps (64
// columns each) of the tile's 256 rows a load, copied by one warp in 16-byte asynchronous copies, neighbouring pieces by
// neighbouring lanes: Q4_K whole super-blocks (144 bytes a row, four steps; rows 144 bytes apart are conflict-free as they
// are), Q8_0 the quants (64 bytes, swizzled), Q6_K the low nibbles (32 bytes, swizzled).  A bulk copy a row instead took
// gate|up of 4096 tokens from 0.87 to 2.08 ms.  What is left (scales, Q6_K's high bits) a thread loads for its own row and
// half, a step ahead.  (Every thread loading its own row's pieces put 16 lines into each request and was the slowest part:
// 0.7 ms of 1.2 for gate|up of 512 experts of 1536 x 3072 with everything else taken out.  TMA tensor loads do not fit: the
// host does not know how many experts there are, and a tensor map that claims more of them than are in memory may not be
// given to the unit; it faulted where memory ends soon after a small matrix.)
// volatile: the loads stay where they are written, a step ahead of their use
__device__ __forceinline__ uint2 mu_ld8(const void* p) {
    uint2 v;
    asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned mu_ld2(const void* p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
template <int TYPE> struct MuRaw {   // Q8_0, Q6_K
    static constexpr int STEPS = 1, WIDTH = TYPE == FNX_Q8_0 ? 64 : 32, SLOTS = 4;
    static __device__ __forceinline__ int row_bytes(const MuArgs& a) { return TYPE == FNX_Q8_0 ? a.ncols : a.ncols / 2; }
    static __device__ __forceinline__ size_t expert_bytes(const MuArgs& a) { return TYPE == FNX_Q8_0 ? a.stride : a.stride * 16; }
    static __device__ __forceinline__ int swizzle(int row) { return TYPE == FNX_Q8_0 ? (row >> 1) & 3 : (row >> 2) & 1; }   // of a row's pieces
    uint4 q0, q1;   // Q8_0: the 32 quants; Q6_K: q0 = low nibbles, q1.xy = high bits
    unsigned s, d;  // Q8_0: s = scale; Q6_K: s = the two scales, d = d
    __device__ __forceinline__ void fetch(const MuArgs& a, int expert, int row, int half, int step) {
        const int k0 = step * MU_KC;
        if (32 * half >= a.ncols - k0) return;   // a last tile of 32 columns
        if (TYPE == FNX_Q8_0) {
            s = mu_ld2(reinterpret_cast<const uint16_t*>(a.b + (size_t) expert * a.stride_b) + (size_t) row * (a.ncols / 32) + k0 / 32 + half);
        } else {
            const size_t g = (size_t) expert * a.stride + (size_t) row * (a.ncols / 32) + k0 / 32 + half;
            const uint2 h = mu_ld8(reinterpret_cast<const uint2*>(a.b) + g);
            q1.x = h.x, q1.y = h.y;
            s = mu_ld2(reinterpret_cast<const uint16_t*>(a.c) + g);
            d = mu_ld2(reinterpret_cast<const uint16_t*>(a.d) + g);
        }
    }
    __device__ __forceinline__ void begin(const unsigned char*, int) {}
    __device__ __forceinline__ void read(const unsigned char* slot, int row, int half, int) {
        if (TYPE == FNX_Q8_0) {
            const uint4* r = reinterpret_cast<const uint4*>(slot + row * 64);
            q0 = r[(2 * half) ^ swizzle(row)], q1 = r[(2 * half + 1) ^ swizzle(row)];
        } else {
            q0 = reinterpret_cast<const uint4*>(slot + row * 32)[half ^ swizzle(row)];
        }
    }
};
template <> struct MuRaw<FNX_Q4_K> {
    static constexpr int STEPS = 4, WIDTH = 144, SLOTS = 2;
    static __device__ __forceinline__ int row_bytes(const MuArgs& a) { return a.ncols / 256 * 144; }
    static __device__ __forceinline__ size_t expert_bytes(const MuArgs& a) { return a.stride; }
    static __device__ __forceinline__ int swizzle(int) { return 0; }
    uint4 hd, q[4];
    __device__ __forceinline__ void fetch(const MuArgs&, int, int, int, int) {}
    __device__ __forceinline__ void begin(const unsigned char* slot, int row) { hd = *reinterpret_cast<const uint4*>(slot + row * 144); }
    __device__ __forceinline__ void read(const unsigned char* slot, int row, int half, int j) {
        q[j] = *reinterpret_cast<const uint4*>(slot + row * 144 + 16 + 32 * j + 16 * half);
    }
};

// 8 consecutive f16 values of row `row` at 16-byte piece `chunk` of the 128-byte row
__device__ __forceinline__ void mu_put(unsigned tile, int row, int chunk, __half2 v0, __half2 v1, __half2 v2, __half2 v3) {
    const unsigned at = tile + row * 128 + ((chunk ^ (row & 7)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(mu_u(v0)), "r"(mu_u(v1)), "r"(mu_u(v2)), "r"(mu_u(v3)) : "memory");
}

// tile j of the raw set (j < STEPS) into the A operand's stage
__device__ __forceinline__ void mu_dequant(const MuRaw<FNX_Q4_K>& r, int j, unsigned tile, int row, int half) {
    // byte l of the 16: value 16 half + l of sub-block 2 j (low nibble) and of sub-block 2 j + 1 (high nibble)
    const float d = h2f((uint16_t) (r.hd.x & 0xffff)), dmin = h2f((uint16_t) (r.hd.x >> 16));
    float sc0, m0, sc1, m1;
    q4k_scale_min_pair(r.hd, j, sc0, m0, sc1, m1);
    const __half2 d0 = __float2half2_rn(fmul(d, sc0)), n0 = __float2half2_rn(-fmul(dmin, m0));
    const __half2 d1 = __float2half2_rn(fmul(d, sc1)), n1 = __float2half2_rn(-fmul(dmin, m1));
    const __half2 k = mu_h2(0x6400);
    const unsigned q[4] = {r.q[j].x, r.q[j].y, r.q[j].z, r.q[j].w};
    __half2 lo[8], hi[8];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        __half2 u, v;
        mu_bytes(q[w] & 0x0F0F0F0Fu, k, u, v);
        lo[2 * w] = __hfma2(u, d0, n0), lo[2 * w + 1] = __hfma2(v, d0, n0);
        mu_bytes((q[w] >> 4) & 0x0F0F0F0Fu, k, u, v);
        hi[2 * w] = __hfma2(u, d1, n1), hi[2 * w + 1] = __hfma2(v, d1, n1);
    }
    mu_put(tile, row, 2 * half, lo[0], lo[1], lo[2], lo[3]);
    mu_put(tile, row, 2 * half + 1, lo[4], lo[5], lo[6], lo[7]);
    mu_put(tile, row, 4 + 2 * half, hi[0], hi[1], hi[2], hi[3]);
    mu_put(tile, row, 5 + 2 * half, hi[4], hi[5], hi[6], hi[7]);
}
__device__ __forceinline__ void mu_dequant(const MuRaw<FNX_Q8_0>& r, int, unsigned tile, int row, int half) {
    // the signed quants offset by 128 become bytes 0..255: 1024 + 128 + q, less 1152
    const __half2 d = mu_h2((unsigned short) r.s), k = mu_h2(0x6480);
    const unsigned q[8] = {r.q0.x, r.q0.y, r.q0.z, r.q0.w, r.q1.x, r.q1.y, r.q1.z, r.q1.w};
    __half2 y[16];
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        __half2 u, v;
        mu_bytes(q[w] ^ 0x80808080u, k, u, v);
        y[2 * w] = __hmul2(u, d), y[2 * w + 1] = __hmul2(v, d);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) mu_put(tile, row, 4 * half + c, y[4 * c], y[4 * c + 1], y[4 * c + 2], y[4 * c + 3]);
}
__device__ __forceinline__ void mu_dequant(const MuRaw<FNX_Q6_K>& r, int, unsigned tile, int row, int half) {
    // a unit: byte i of the 16 holds value i (low nibble) and value 16 + i (high nibble); the two high bits of value
    // 4 w + b sit in byte (w / 4) 4 + b of the 8 at bit 2 (w % 4); codes 0..63 less 32; scale 0 for values < 16
    const float d = h2f((uint16_t) r.d);
    const int s0 = (int) (signed char) (r.s & 0xff), s1 = (int) (signed char) ((r.s >> 8) & 0xff);
    const __half2 d0 = __float2half2_rn(fmul(d, (float) s0)), d1 = __float2half2_rn(fmul(d, (float) s1));
    const __half2 k = mu_h2(0x6420);   // 1024 + 32
    const unsigned q[4] = {r.q0.x, r.q0.y, r.q0.z, r.q0.w};
    __half2 lo[8], hi[8];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        __half2 u, v;
        mu_bytes((q[w] & 0x0F0F0F0Fu) | (((r.q1.x >> (2 * w)) & 0x03030303u) << 4), k, u, v);
        lo[2 * w] = __hmul2(u, d0), lo[2 * w + 1] = __hmul2(v, d0);
        mu_bytes(((q[w] >> 4) & 0x0F0F0F0Fu) | (((r.q1.y >> (2 * w)) & 0x03030303u) << 4), k, u, v);
        hi[2 * w] = __hmul2(u, d1), hi[2 * w + 1] = __hmul2(v, d1);
    }
    mu_put(tile, row, 4 * half, lo[0], lo[1], lo[2], lo[3]);
    mu_put(tile, row, 4 * half + 1, lo[4], lo[5], lo[6], lo[7]);
    mu_put(tile, row, 4 * half + 2, hi[0], hi[1], hi[2], hi[3]);
    mu_put(tile, row, 4 * half + 3, hi[4], hi[5], hi[6], hi[7]);
}

// The first jobs of the pairs among jobs [base, base + cnt), cnt <= MU_LIST, in order; all threads.  An expert's jobs are
// consecutive and are paired from its first one; `run`: where the run of the job before `base` began.
__device__ int mu_list_pairs(const FnxBigJob* jobs, int base, int cnt, int& run, uint16_t* list) {
    __shared__ int wstart[MU_THREADS / 32], wcount[MU_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int per = (cnt + MU_THREADS - 1) / MU_THREADS, lo = base + min(cnt, tid * per), hi = base + min(cnt, (tid + 1) * per);
    int start = -1;   // the last run that begins among this thread's jobs
    for (int j = lo; j < hi; ++j)
        if (j == 0 || jobs[j].w != jobs[j - 1].w) start = j;
    int before = start;   // the last run that begins at or before this thread's jobs
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before = max(before, v);
    }
    if (lane == 31) wstart[warp] = before;
    before = __shfl_up_sync(0xffffffffu, before, 1);
    if (lane == 0) before = -1;
    __syncthreads();
    int last = run;
    for (int w = 0; w < MU_THREADS / 32; ++w) {
        if (w < warp) before = max(before, wstart[w]);
        last = max(last, wstart[w]);
    }
    before = max(before, run);
    auto is_first = [&](int j, int& at) {
        if (j == 0 || jobs[j].w != jobs[j - 1].w) at = j;
        return ((j - at) & 1) == 0;
    };
    int n = 0, at = before;
    for (int j = lo; j < hi; ++j) n += is_first(j, at);
    int pre = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += v;
    }
    if (lane == 31) wcount[warp] = pre;
    __syncthreads();
    int total = 0;
    pre -= n;
    for (int w = 0; w < MU_THREADS / 32; ++w) {
        if (w < warp) pre += wcount[w];
        total += wcount[w];
    }
    at = before;
    for (int j = lo; j < hi; ++j)
        if (is_first(j, at)) list[pre++] = (uint16_t) (j - base);
    run = last;
    __syncthreads();
    return total;
}

// out[jb.out[j] * nrows + row] = sum_k W_e[row][k] x[jb.y[j] * ncols + k]
template <int TYPE>
__global__ void __launch_bounds__(MU_THREADS, 1) k_moe_umma(const MuArgs a) {
    using Raw = MuRaw<TYPE>;
    const int tid = threadIdx.x, warp = (int) um_uniform(tid >> 5), lane = tid & 31;
    const int njobs = min(*a.njobs, a.njobs_cap);
    extern __shared__ __align__(1024) unsigned char mu_smem[];
    // the swizzle is a function of the shared-memory address: operand tiles start on 1024-byte boundaries
    unsigned char* stages = mu_smem + ((1024u - (um_s32(mu_smem) & 1023u)) & 1023u);
    unsigned char* raw = stages + (size_t) MU_NS * MU_STAGE;
    uint16_t* list = reinterpret_cast<uint16_t*>(raw + MU_RAW);
    static_assert(MU_COPY == 2 * MU_NS, "two copy warps a stage");
    static_assert(Raw::SLOTS * Raw::WIDTH * MU_BM <= MU_RAW, "the raw ring");
    __shared__ __align__(8) unsigned long long full[MU_NS], empty[MU_NS], done[2], freed[2], idle, rfull[Raw::SLOTS], rempty[Raw::SLOTS];
    __shared__ unsigned tmem_base;
    __shared__ int ys[MU_COPY][MU_NMAX / 2];   // a copy warp's rows of x, -1: none
    if (tid == 0) {
        for (int s = 0; s < MU_NS; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(um_s32(&full[s])), "r"(MU_PROD / 32 + 64));   // the producers' warps and two copy warps' lanes
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(um_s32(&empty[s])));
        }
        for (int s = 0; s < Raw::SLOTS; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 32;" ::"r"(um_s32(&rfull[s])));   // the loader's lanes
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(um_s32(&rempty[s])), "r"(MU_PROD / 32));
        }
        for (int s = 0; s < 2; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(um_s32(&done[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(um_s32(&freed[s])), "r"(MU_PROD / 32));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(um_s32(&idle)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MU_PROD / 32) {   // all 512 columns of tensor memory: two results of 2 x 128 rows x (64 + 64)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(um_s32(&tmem_base)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // a last step of 32 columns (an FF slice of 96) fills half a stage: two MMAs instead of four
    const int nk = (a.ncols + MU_KC - 1) / MU_KC, ntiles = (a.nrows + MU_BM - 1) / MU_BM;
    const unsigned st_s = um_s32(stages);
    bool alive = true;   // false after a wait ran out
    unsigned g0 = 0, seq = 0, rc = 0;   // steps, tiles and raw loads that this role has behind it
    CopyRing<Raw::SLOTS> ring;          // the loader's side of the raw loads
    const int nsteps = (nk + Raw::STEPS - 1) / Raw::STEPS;
    int run = 0;
    for (int base = 0; base < njobs; base += MU_LIST) {
        const int items = mu_list_pairs(a.jobs, base, min(MU_LIST, njobs - base), run, list) * ntiles;
        const int first = blockIdx.x, stride = gridDim.x;
        auto job_of = [&](int it) { return base + list[it / ntiles]; };
        // a tile's jobs' rows; n2: the partner's, 0 without one
        auto rows_of = [&](int ji, int& n, int& n2) {
            n = min(max(a.jobs[ji].n, 0), FNX_PF_JOB);
            const bool paired = ji + 1 < njobs && a.jobs[ji + 1].w == a.jobs[ji].w;
            n2 = paired ? min(max(a.jobs[ji + 1].n, 0), FNX_PF_JOB) : 0;
        };
        auto cols_of = [&](int n, int n2) { return n2 ? FNX_PF_JOB + 16 * ((n2 + 15) / 16) : 16 * ((n + 15) / 16); };   // N of the MMAs
        if (warp < MU_PROD / 32) {
            // ---- producers: warp w owns rows 16 w .. + 15 of the tile, lanes 0..15 the first 32 columns of a step and lanes
            // 16..31 the last 32 (the two lanes of a row read neighbouring bytes: a warp's load touches 16 lines, and a
            // quarter-warp's stores 8 different rows of one 16-byte column: no bank conflicts)
            const int row = 16 * warp + (lane & 15), half = lane >> 4;
            auto wrow = [&](int it) { return min(it % ntiles * MU_BM + row, a.nrows - 1); };   // rows past the matrix repeat the last one; never written out
            // the result of tile number t, item `it`, out of tensor memory: warp w reads lanes 32 (w % 4) .. + 31 (its quarter)
            // of the rows' lower or upper 128, the first or second half of the columns; 32 lanes write 32 consecutive floats
            auto write_out = [&](int it, unsigned t) {
                const unsigned buf = t & 1u;
                const int ji = job_of(it);
                int n, n2;
                rows_of(ji, n, n2);
                if (alive) alive = um_wait(&done[buf], (t >> 1) & 1u, a.fault);
                const bool ok = __all_sync(0xffffffffu, alive);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int hi = (warp >> 2) & 1, orow = it % ntiles * MU_BM + 128 * hi + 32 * (warp & 3) + lane;
                const int cols = cols_of(n, n2) / 2, c0 = (warp >> 3) * cols;
                if (ok)
                    for (int c = c0; c < c0 + cols; c += 8) {
                        unsigned v[8];
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                                     : "r"(tmem_base + ((unsigned) (32 * (warp & 3)) << 16) + buf * 256u + 128u * hi + (unsigned) c));
                        const bool second = c >= FNX_PF_JOB;
                        const int jj = c & (FNX_PF_JOB - 1), live = second ? n2 : n;
                        const int4* op = reinterpret_cast<const int4*>(a.jobs[ji + second].out + jj);
                        int o[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) o[i] = reinterpret_cast<const int*>(op)[i];
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (jj + i < live && orow < a.nrows) a.out[(size_t) o[i] * a.nrows + orow] = __uint_as_float(v[i]);
                    }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mu_arrive(&freed[buf]);
            };
            Raw cur, nxt;
            if (first < items) cur.fetch(a, a.jobs[job_of(first)].w, wrow(first), half, 0);
            int prev = -1;
            for (int it = first; it < items; it += stride, ++seq, g0 += nk) {
                const int expert = a.jobs[job_of(it)].w, wr = wrow(it);
                const bool more = it + stride < items;
                const int nexpert = more ? a.jobs[job_of(it + stride)].w : 0, nwr = more ? wrow(it + stride) : 0;
#pragma unroll 1
                for (int sidx = 0; sidx < nsteps; ++sidx, ++rc) {
                    if (sidx + 1 < nsteps) nxt.fetch(a, expert, wr, half, sidx + 1);
                    else if (more) nxt.fetch(a, nexpert, nwr, half, 0);
                    const unsigned slot = rc % Raw::SLOTS;
                    const unsigned char* rs = raw + slot * (Raw::WIDTH * MU_BM);
                    if (alive) alive = um_wait(&rfull[slot], (rc / Raw::SLOTS) & 1u, a.fault);
                    cur.begin(rs, row);
#pragma unroll
                    for (int j = 0; j < Raw::STEPS; ++j) {
                        const int k = sidx * Raw::STEPS + j;
                        if (k < nk) {
                            const unsigned g = g0 + k, s = g % MU_NS;
                            cur.read(rs, row, half, j);
                            if (g >= MU_NS && alive) alive = um_wait(&empty[s], (g / MU_NS - 1) & 1u, a.fault);
                            if (32 * half < a.ncols - k * MU_KC) mu_dequant(cur, j, st_s + s * MU_STAGE + (row >> 7) * 16384, row & 127, half);
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes before the tensor core's reads
                            __syncwarp();
                            if (lane == 0) mu_arrive(&full[s]);
                        }
                    }
                    if (lane == 0) mu_arrive(&rempty[slot]);   // every lane's reads lie before the last step's warp barrier
                    cur = nxt;
                    if (prev >= 0 && ((sidx + 1) * Raw::STEPS >= MU_NS - 1 || sidx + 1 == nsteps)) {
                        write_out(prev, seq - 1);
                        prev = -1;
                    }
                }
                prev = it;
            }
            if (prev >= 0) write_out(prev, seq - 1);
        } else if (warp == MU_PROD / 32 + 1) {
            // ---- the raw weights' copies, as far ahead as the ring holds, across the ends of tiles.  Rows past the matrix repeat
            // the last one, pieces past a row's end are left out: nothing is read that is not the matrix's
            const auto landed = [&](unsigned s, unsigned parity) { return um_wait(&rfull[s], parity, a.fault); };
            const auto used = [&](unsigned s, unsigned parity) { return um_wait(&rempty[s], parity, a.fault); };
            const int row_bytes = Raw::row_bytes(a);
            unsigned off[9];   // Q4_K: this lane's pieces among 32 rows
            if (TYPE == FNX_Q4_K) {
#pragma unroll
                for (int k = 0; k < 9; ++k) off[k] = (unsigned) ((lane + 32 * k) / 9 * row_bytes + (lane + 32 * k) % 9 * 16);
            }
            for (int it = first; it < items && ring.alive; it += stride) {
                const int expert = a.stride ? a.jobs[job_of(it)].w : 0;   // stride 0: one matrix for all
                const unsigned char* src = a.a + (size_t) expert * Raw::expert_bytes(a);
                const int row0 = it % ntiles * MU_BM, last = a.nrows - 1 - row0;
                src += (size_t) row0 * row_bytes;
                for (int c = 0; c < nsteps; ++c) {
                    ring.alive = __all_sync(0xffffffffu, ring.acquire(used, landed));
                    if (!ring.alive) break;
                    const unsigned dst = um_s32(raw + ring.slot * (Raw::WIDTH * MU_BM));
                    const unsigned char* from = src + c * Raw::WIDTH;
                    if constexpr (TYPE == FNX_Q4_K) {   // nine pieces a row, one after the other in the slot: 32 rows every nine pieces of a lane
                        const unsigned to = dst + 16 * lane;
                        if (last >= MU_BM - 1) {
                            const unsigned char* q = from;
#pragma unroll
                            for (int b = 0; b < MU_BM / 32; ++b, q += 32 * row_bytes)
#pragma unroll
                                for (int k = 0; k < 9; ++k)
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (9 * b + k) * 512), "l"(q + off[k]));
                        } else {
#pragma unroll 4
                            for (int i = 0; i < MU_BM * 9 / 32; ++i) {
                                const int e = lane + 32 * i;
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 512 * i),
                                             "l"(from + (size_t) (unsigned) (min(e / 9, last) * row_bytes + 16 * (e % 9))));
                            }
                        }
                    } else {   // a lane the same piece of every 32 / PC-th row (the swizzle is the same for all of them)
                        constexpr int PC = Raw::WIDTH / 16, RP = 32 / PC;
                        const int r0 = lane / PC, pc = lane % PC;
                        const unsigned to = dst + r0 * Raw::WIDTH + ((pc ^ Raw::swizzle(r0)) << 4);
                        if (c * Raw::WIDTH + 16 * pc < row_bytes) {
                            if (last >= MU_BM - 1) {
                                const unsigned char* q = from + r0 * row_bytes + 16 * pc;
                                const int step = RP * row_bytes;
#pragma unroll
                                for (int i = 0; i < MU_BM / RP; ++i, q += step)
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * RP * Raw::WIDTH), "l"(q));
                            } else {
#pragma unroll 4
                                for (int i = 0; i < MU_BM / RP; ++i)
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i * RP * Raw::WIDTH),
                                                 "l"(from + (size_t) (unsigned) (min(r0 + RP * i, last) * row_bytes + 16 * pc)));
                            }
                        }
                    }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(um_s32(&rfull[ring.slot])) : "memory");
                    ring.asked();
                }
            }
        } else if (warp > MU_PROD / 32) {
            // ---- the activation rows, by asynchronous copies, two warps a step in turn: every stage's copies are issued side by side.  Lane i takes
            // the 16-byte piece i % 8 of rows i / 8 (+ 4 in the second warp), + 8, ... of the stage's 128 (0..63 the job's, 64..127 its partner's)
            const unsigned mine = (warp - MU_PROD / 32 - 2) >> 1;
            const int xc = lane & 7, r0 = (lane >> 3) + 4 * ((warp - MU_PROD / 32) & 1);
            for (int it = first; it < items; it += stride, g0 += nk) {
                const int ji = job_of(it);
                int n, n2;
                rows_of(ji, n, n2);
                const FnxBigJob &jb = a.jobs[ji], &jb2 = a.jobs[n2 ? ji + 1 : ji];
                __syncwarp();
                int* yw = ys[warp - MU_PROD / 32 - 2];   // [i][lane / 8]: row r0 + 8 i
                for (int q = lane; q < MU_NMAX / 2; q += 32) {   // the rows' indices, for every step of the tile
                    const int j = (q & 3) + 4 * ((warp - MU_PROD / 32) & 1) + 8 * (q >> 2);
                    yw[q] = j < FNX_PF_JOB ? (j < n ? jb.y[j] : -1) : (j - FNX_PF_JOB < n2 ? jb2.y[j - FNX_PF_JOB] : -1);
                }
                __syncwarp();
#pragma unroll 1
                for (int k = (int) ((mine + MU_NS - g0 % MU_NS) % MU_NS); k < nk; k += MU_NS) {
                    const unsigned g = g0 + k, s = g % MU_NS;
                    if (g >= MU_NS && alive) alive = um_wait(&empty[s], (g / MU_NS - 1) & 1u, a.fault);
                    const unsigned tile = st_s + s * MU_STAGE + MU_ABYTES;
                    const uint16_t* xk = a.x + (size_t) k * MU_KC + 8 * xc;
                    if (8 * xc < a.ncols - k * MU_KC) {
#pragma unroll 4
                        for (int j = r0; j < (n2 ? FNX_PF_JOB + n2 : n); j += 8) {
                            const int y = yw[(j >> 3) * 4 + (lane >> 3)];
                            if (y >= 0)
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tile + j * 128 + ((xc ^ (j & 7)) << 4)), "l"(xk + (size_t) y * a.ncols));
                        }
                    }
                    // the lane's arrival, made by the copies' unit when they have landed (the issuing warp fences them)
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(um_s32(&full[s])) : "memory");
                }
            }
        } else {
            // ---- the issuing warp: a stage's MMAs once it is full; the commit frees the stage
            for (int it = first; it < items; it += stride, ++seq, g0 += nk) {
                int n, n2;
                rows_of(job_of(it), n, n2);
                const unsigned idesc = (1u << 4) | ((unsigned) (cols_of(n, n2) >> 3) << 17) | ((128u >> 4) << 24);   // D f32, A and B f16 K-major
                const unsigned d = um_uniform(tmem_base) + (seq & 1u) * 256u;
                const bool upper = it % ntiles * MU_BM + 128 < a.nrows;
                if (seq >= 2 && alive) alive = um_wait(&freed[seq & 1u], ((seq >> 1) - 1) & 1u, a.fault);
#pragma unroll 1
                for (int k = 0; k < nk; ++k) {
                    const unsigned g = g0 + k, s = g % MU_NS;
                    if (alive) alive = um_wait(&full[s], (g / MU_NS) & 1u, a.fault);
                    alive = __all_sync(0xffffffffu, alive);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the copied rows before the tensor core's reads
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (um_elect()) {
                        const unsigned long long da = um_desc(st_s + s * MU_STAGE), db = um_desc(st_s + s * MU_STAGE + MU_ABYTES);
                        const int steps = min(MU_KC, a.ncols - k * MU_KC) / 16;
#pragma unroll
                        for (int ks = 0; ks < MU_KC / 16; ++ks)
                            if (ks < steps) {
                                um_mma(d, da + 2 * ks, db + 2 * ks, idesc, (unsigned) (k | ks));
                                if (upper) um_mma(d + 128, da + 1024 + 2 * ks, db + 2 * ks, idesc, (unsigned) (k | ks));   // 128 rows on: 16 384 bytes
                            }
                        um_commit(&empty[s]);
                    }
                    __syncwarp();
                }
                if (um_elect()) um_commit(&done[seq & 1u]);
                __syncwarp();
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // only a wait that ran out leaves copies in flight here
        __syncthreads();   // the list may be rewritten
    }
    if (warp == MU_PROD / 32) {   // the results' readers waited for the MMAs, unless a wait of theirs ran out
        if (um_elect()) um_commit(&idle);
        __syncwarp();
        um_wait(&idle, 0u, a.fault);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MU_PROD / 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
}

// h = silu(gate) * up of the stacked rows, rounded to f16 (reference src/moe_mma.cuh:381-388)
__global__ void __launch_bounds__(256) k_swiglu_h16(const float* __restrict__ gu, int ffs, size_t total, uint16_t* __restrict__ h) {
    for (size_t e = (size_t) blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t) gridDim.x * 256) {
        const size_t r = e / ffs, i = e % ffs;
        const float g = gu[r * 2 * ffs + i];
        h[e] = f2h(fmul(ex_silu(g), gu[r * 2 * ffs + ffs + i]));
    }
}

// the same for rows of whole 16-byte pieces: eight values a thread, in flight together.  Bound by HBM (10 bytes a value); a
// value a thread with a 64-bit division each ran at 2.0 TB/s (40 960 rows of 768: 157 us, now 59).
__global__ void __launch_bounds__(256) k_swiglu_h16_v8(const float4* __restrict__ gu, unsigned f8, unsigned total, uint4* __restrict__ h) {
    const unsigned e = blockIdx.x * 256 + threadIdx.x;
    if (e >= total) return;
    const unsigned r = e / f8, i = e - r * f8;
    const float4* g = gu + (size_t) r * 4 * f8 + 2 * i;
    const float4 g0 = __ldcs(g), g1 = __ldcs(g + 1), u0 = __ldcs(g + 2 * f8), u1 = __ldcs(g + 2 * f8 + 1);
    const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    unsigned o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        o[k] = f2h(fmul(ex_silu(gv[2 * k]), uv[2 * k])) | (unsigned) f2h(fmul(ex_silu(gv[2 * k + 1]), uv[2 * k + 1])) << 16;
    h[e] = make_uint4(o[0], o[1], o[2], o[3]);
}

static int moe_umma(const char* what, const FnxExperts* A, const FnxBigJob* jobs, const int* njobs, int njobs_cap, const uint16_t* x, float* out,
                    cudaStream_t st) {
    FNX_REQUIRE(A && jobs && njobs && njobs_cap >= 1 && x && out, "%s: no experts, jobs, rows or output", what);
    FNX_REQUIRE(A->nrows >= 1 && A->ncols >= 32 && A->ncols % 32 == 0, "%s: %d x %d (columns in units of 32)", what, A->nrows, A->ncols);
    FNX_REQUIRE(((uintptr_t) x % 16) == 0, "%s: activation rows not 16-byte aligned", what);
    unsigned* fault = device_fault_word();
    FNX_REQUIRE(fault, "%s: no device fault word (no current device?)", what);
    MuArgs a{A->type, A->nrows, A->ncols, (const unsigned char*) A->a, (const unsigned char*) A->b, (const unsigned char*) A->c,
             (const unsigned char*) A->d, A->stride, A->stride_b, jobs, njobs, njobs_cap, x, out, fault};
    int dev = 0, nsm = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return fail("%s: no device", what);
    const int grid = (int) std::min<long long>(nsm, (long long) ((A->nrows + MU_BM - 1) / MU_BM) * njobs_cap);
#define MU_LAUNCH(T)                                                            \
    if (smem_optin(k_moe_umma<T>, MU_SMEM, what)) return 1;                     \
    k_moe_umma<T><<<grid, MU_THREADS, MU_SMEM, st>>>(a);                        \
    return launch_ok(what);
    if (A->type == FNX_Q4_K) {
        FNX_REQUIRE(A->ncols % 256 == 0 && ((uintptr_t) A->a % 16) == 0 && A->stride % 16 == 0, "%s q4_K: %d columns, rows 16-byte aligned", what, A->ncols);
        MU_LAUNCH(FNX_Q4_K)
    }
    if (A->type == FNX_Q8_0) {
        FNX_REQUIRE(((uintptr_t) A->a % 16) == 0 && A->stride % 16 == 0 && A->stride_b % 2 == 0, "%s q8_0: planes 16-byte aligned", what);
        MU_LAUNCH(FNX_Q8_0)
    }
    if (A->type == FNX_Q6_K) {
        FNX_REQUIRE(((uintptr_t) A->a % 16) == 0 && ((uintptr_t) A->b % 8) == 0, "%s q6_K: unit planes not aligned", what);
        MU_LAUNCH(FNX_Q6_K)
    }
#undef MU_LAUNCH
    return fail("%s: expert type %d not supported (Q4_K, Q8_0, Q6_K units)", what, A->type);
}

}  // namespace fnxk

using namespace fnxk;

extern "C" {

int fnx_moe_gate_up_mma(const FnxExperts* A, const FnxBigJob* jobs, const int* njobs, int njobs_cap, const uint16_t* xh, float* gu, void* st) {
    return moe_umma("moe_gate_up_mma", A, jobs, njobs, njobs_cap, xh, gu, strm(st));
}

int fnx_swiglu_h16(const float* gu, int ffs, int P, uint16_t* h16, void* st) {
    FNX_REQUIRE(gu && h16 && ffs >= 1 && P >= 0, "swiglu_h16: %d rows of %d", P, ffs);
    if (!P) return 0;
    const size_t total = (size_t) P * ffs;
    if (ffs % 8 == 0 && (uintptr_t) gu % 16 == 0 && (uintptr_t) h16 % 16 == 0 && total / 8 < (1ull << 31)) {
        const unsigned pieces = (unsigned) (total / 8);
        k_swiglu_h16_v8<<<(pieces + 255) / 256, 256, 0, strm(st)>>>((const float4*) gu, ffs / 8, pieces, (uint4*) h16);
        return launch_ok("swiglu_h16");
    }
    k_swiglu_h16<<<(unsigned) std::min<size_t>(4096, (total + 255) / 256), 256, 0, strm(st)>>>(gu, ffs, total, h16);
    return launch_ok("swiglu_h16");
}

int fnx_moe_down_mma(const FnxExperts* A, const FnxBigJob* jobs, const int* njobs, int njobs_cap, const uint16_t* h16, float* part, void* st) {
    return moe_umma("moe_down_mma", A, jobs, njobs, njobs_cap, h16, part, strm(st));
}
}
