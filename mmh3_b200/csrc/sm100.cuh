// Thin wrappers over the Blackwell (sm_100a) instructions the attention kernels are built from:
// mbarrier, TMA tile loads (cp.async.bulk.tensor), tensor memory (TMEM) allocation and access, and
// the tcgen05 UMMA with its shared-memory and instruction descriptors.
//
// Every wait in here is bounded. A wait that runs out records a code in a status word and raises a
// flag in shared memory that every other wait of the CTA polls, so that a broken pipeline drains
// and returns instead of hanging the device.
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace sm100 {

// About one second at the clocks a B200 runs at: far longer than any wait of a healthy pipeline.
constexpr long long WAIT_LIMIT_CYCLES = 2000000000ll;

__device__ __forceinline__ uint32_t smem_u32(const void *pointer) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(pointer));
}

// The warp's index in its CTA, in a form the compiler knows to be the same for all 32 lanes.
__device__ __forceinline__ int warp_index() {
    return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
}

// True in one lane of a converged warp. A role that one thread plays (TMA, MMA) goes inside
// `if (warp == ROLE) if (elect_one())` over a warp_index(): the compiler then knows that a single
// thread gets there, which it cannot tell from `lane == 0`, and keeps the operands of
// tcgen05.mma in uniform registers instead of moving each one there for every instruction. Eight
// MMAs of 128 x 128 x 16 are issued in 143 cycles instead of 400-460, less than the 512 they run
// for, so the tensor cores' queue fills up and the thread's next wait costs them nothing.
__device__ __forceinline__ bool elect_one() {
    uint32_t elected;
    asm volatile("{\n"
                 ".reg .pred p;\n"
                 "elect.sync _|p, 0xffffffff;\n"
                 "selp.u32 %0, 1, 0, p;\n"
                 "}"
                 : "=r"(elected));
    return elected != 0;
}

// ---------------------------------------------------------------------------------------------
// Kernels launched with launch_behind (common.cuh): the next kernel of the stream may be set up
// once every CTA of this one has said so, and waits here for the kernels before it to have finished
// and their writes to be visible, before it touches global memory. Every thread waits, so no kernel
// ends before the ones it was launched behind.
//
// Tensor memory is what CTAs of two kernels on one multiprocessor could wait for each other over: one
// that holds it and waits for the kernel before, one of that kernel that waits in its tcgen05.alloc,
// where no limit ends the wait. So a kernel takes its columns after wait_for_kernels_before, and lets
// the next one begin when it has them, whatever fits beside what.

__device__ __forceinline__ void let_next_kernel_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Returns zero, for the addresses of read-only loads (__ldg, and what the compiler makes one of behind
// a const __restrict__ pointer): the clobber of memory does not hold those back, and what the kernels
// before have written is to be read after the wait.
[[nodiscard]] __device__ __forceinline__ int wait_for_kernels_before() {
    int zero;
    asm volatile("griddepcontrol.wait;\n"
                 "mov.u32 %0, 0;"
                 : "=r"(zero)
                 :
                 : "memory");
    return zero;
}

// ---------------------------------------------------------------------------------------------
// mbarrier

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Makes the initialised barriers visible to the async proxy (TMA, tcgen05.commit).
__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n"
                 ".reg .pred p;\n"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n"
                 "}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

// What a CTA shares about a wait that gave up: a flag in shared memory that its other waits poll,
// and the status word in global memory the host reads.
struct Watchdog {
    volatile uint32_t *abort_flag;
    unsigned int *status;
};

// Waits for the phase of `bar` with parity `parity` to complete. Returns false when the wait ran
// out or another wait of the CTA already had; `code` then says which wait this was.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const Watchdog &watchdog,
                                          unsigned int code) {
    if (mbar_try_wait(bar, parity)) {
        return true;
    }
    const long long start = clock64();
    for (;;) {
        #pragma unroll 1
        for (int spin = 0; spin < 64; spin++) {
            if (mbar_try_wait(bar, parity)) {
                return true;
            }
        }
        if (*watchdog.abort_flag != 0) {
            return false;
        }
        if (clock64() - start > WAIT_LIMIT_CYCLES) {
            *watchdog.abort_flag = 1;
            atomicCAS(watchdog.status, 0u, code);
            return false;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// TMA: one box of a tiled tensor map into shared memory, completing `bar` by its byte count.

__device__ __forceinline__ void tma_load_2d(uint32_t destination, const CUtensorMap *map,
                                            uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%3, %4}], [%2];" ::"r"(destination),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t destination, const CUtensorMap *map,
                                            uint32_t bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(destination),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t destination, const CUtensorMap *map,
                                            uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
                 "[%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(destination),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}

// A hint: the 128-byte line holding `address` into L1.
__device__ __forceinline__ void prefetch_l1(const void *address) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(address));
}

__device__ __forceinline__ void tma_prefetch_descriptor(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Tensor memory

// Allocates `columns` (a power of two, at least 32) TMEM columns and writes their base address to
// shared memory. One whole warp calls it, and the same warp frees the columns.
__device__ __forceinline__ void tmem_alloc(uint32_t destination, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     destination),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns)
                 : "memory");
}

__device__ __forceinline__ void tcgen05_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tcgen05_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Makes `bar` complete once every MMA this thread has issued so far has.
__device__ __forceinline__ void tcgen05_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::
                     "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_wait_load() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_wait_store() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// 32 consecutive 32-bit columns of this thread's TMEM lane (the warp's lane quarter plus the lane
// index), starting at `address`. The registers are valid after tmem_wait_load.
__device__ __forceinline__ void tmem_load_32(uint32_t address, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(address)
        : "memory");
}

__device__ __forceinline__ void tmem_store_32(uint32_t address, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
            address),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
        "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void tmem_store_16(uint32_t address, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
                     address),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
                 "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
                 "r"(r[14]), "r"(r[15])
                 : "memory");
}

__device__ __forceinline__ void tmem_store_8(uint32_t address, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(address),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
                 "r"(r[7])
                 : "memory");
}

// ---------------------------------------------------------------------------------------------
// Pairs of CTAs (clusters of two) on one MMA. A kernel that uses them uses cta_group::2 throughout.

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    return rank;
}

// The address in the cluster of what `address` is in CTA `rank`.
__device__ __forceinline__ uint32_t cluster_address(uint32_t address, uint32_t rank) {
    uint32_t mapped;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(mapped) : "r"(address), "r"(rank));
    return mapped;
}

// Every thread of both CTAs. It has no limit of its own: each CTA gets here because every wait
// before it has one.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
}

// `bar` is a cluster_address.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar)
                 : "memory");
}

// Into this CTA's shared memory, counted by a barrier of either CTA of the pair (`bar` is a
// cluster_address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t destination, const CUtensorMap *map,
                                                 uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 ".cta_group::2 [%0], [%1, {%3, %4}], [%2];" ::"r"(destination),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t destination, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     destination),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc_pair(uint32_t base, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns)
                 : "memory");
}

// Makes `bar` of both CTAs complete once every pair MMA this thread has issued so far has.
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster"
                 ".multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}

// ---------------------------------------------------------------------------------------------
// UMMA descriptors

// Shared-memory matrix descriptor of a tile in the 128-byte swizzle TMA writes (rows of 128 bytes,
// eight rows to a 1024-byte swizzle atom). `leading` and `stride` are byte offsets:
//
// - K-major operand (the contraction runs along a row): `stride` is the distance between groups
//   of eight rows, and `leading` is not used.
// - MN-major operand (the contraction runs down the rows): `stride` is the distance between
//   groups of eight rows of the contraction, and `leading` the distance between slabs of 128
//   bytes (64 16-bit elements) along M or N.
//
// `swizzle` is the layout code of the descriptor: SWIZZLE_128B for rows of 128 bytes, SWIZZLE_64B
// for rows of 64 bytes (eight rows to a 512-byte atom).
constexpr uint64_t SWIZZLE_128B = 2, SWIZZLE_64B = 4;

__device__ __forceinline__ uint64_t smem_descriptor(uint32_t address, uint32_t leading,
                                                    uint32_t stride,
                                                    uint64_t swizzle = SWIZZLE_128B) {
    uint64_t descriptor = 0;
    descriptor |= static_cast<uint64_t>((address >> 4) & 0x3fffu);
    descriptor |= static_cast<uint64_t>((leading >> 4) & 0x3fffu) << 16;
    descriptor |= static_cast<uint64_t>((stride >> 4) & 0x3fffu) << 32;
    descriptor |= 1ull << 46; // descriptor version of sm_100
    descriptor |= swizzle << 61;
    return descriptor;
}

// The same descriptor `bytes` further on in shared memory: the address field is the low 14 bits, in
// units of 16 bytes, and shared memory is smaller than the field, so the addition never carries
// into the next field. The MMA-issuing thread builds each tile's descriptor once and steps through
// it with this, which keeps its instruction stream short.
__device__ __forceinline__ uint64_t advance_descriptor(uint64_t descriptor, uint32_t bytes) {
    return descriptor + (bytes >> 4);
}

// Operand formats of the instruction descriptor.
constexpr uint32_t FORMAT_F16 = 0, FORMAT_BF16 = 1;   // kind::f16
constexpr uint32_t FORMAT_U8 = 0, FORMAT_S8 = 1;      // kind::i8
constexpr uint32_t FORMAT_E4M3 = 0, FORMAT_E5M2 = 1;  // kind::f8f6f4
constexpr uint32_t ACCUMULATE_F16 = 0, ACCUMULATE_F32 = 1, ACCUMULATE_S32 = 2;

// Instruction descriptor of a dense M × N UMMA. A major flag of one says the operand is MN-major.
__host__ __device__ constexpr uint32_t instruction_descriptor(uint32_t accumulator, uint32_t a_format,
                                          uint32_t b_format, uint32_t a_mn_major,
                                          uint32_t b_mn_major, uint32_t m, uint32_t n) {
    return (accumulator << 4) | (a_format << 7) | (b_format << 10) | (a_mn_major << 15) |
           (b_mn_major << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// D (TMEM) = A (smem) · B (smem), or D += A · B when `accumulate` is nonzero. One thread issues it.
#define MMH3_DEFINE_MMA(GROUP, KIND, NAME)                                                        \
    __device__ __forceinline__ void NAME##_ss(uint32_t d, uint64_t a, uint64_t b,                 \
                                              uint32_t instruction, uint32_t accumulate) {        \
        asm volatile("{\n"                                                                        \
                     ".reg .pred p;\n"                                                            \
                     "setp.ne.b32 p, %4, 0;\n"                                                    \
                     "tcgen05.mma." GROUP ".kind::" KIND " [%0], %1, %2, %3, p;\n"                \
                     "}" ::"r"(d),                                                                \
                     "l"(a), "l"(b), "r"(instruction), "r"(accumulate)                            \
                     : "memory");                                                                 \
    }                                                                                             \
    /* The same with A in tensor memory at `a`. */                                                \
    __device__ __forceinline__ void NAME##_ts(uint32_t d, uint32_t a, uint64_t b,                 \
                                              uint32_t instruction, uint32_t accumulate) {        \
        asm volatile("{\n"                                                                        \
                     ".reg .pred p;\n"                                                            \
                     "setp.ne.b32 p, %4, 0;\n"                                                    \
                     "tcgen05.mma." GROUP ".kind::" KIND " [%0], [%1], %2, %3, p;\n"              \
                     "}" ::"r"(d),                                                                \
                     "r"(a), "l"(b), "r"(instruction), "r"(accumulate)                            \
                     : "memory");                                                                 \
    }

MMH3_DEFINE_MMA("cta_group::1", "f16", mma_f16)
MMH3_DEFINE_MMA("cta_group::1", "i8", mma_i8)
MMH3_DEFINE_MMA("cta_group::1", "f8f6f4", mma_f8)
// The same over a pair of CTAs, issued by one thread of the pair's first: M = 256, each CTA with
// 128 rows of A and of D and half of B's rows, at the same places of its own memories.
MMH3_DEFINE_MMA("cta_group::2", "f16", mma_f16_pair)
MMH3_DEFINE_MMA("cta_group::2", "i8", mma_i8_pair)
#undef MMH3_DEFINE_MMA

// Moves registers between the warpgroups of a CTA: every warp of a warpgroup (four consecutive
// warps) executes the same one.
template <int REGISTERS> __device__ __forceinline__ void register_increase() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGISTERS));
}

template <int REGISTERS> __device__ __forceinline__ void register_decrease() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGISTERS));
}

// 32 rows of DIM 16-bit values on their way from a warp that holds a row per lane to global memory,
// through a corner of shared memory of the warp's own (32 * DIM * 2 bytes, on 16 bytes), so that a
// store covers whole rows instead of 16 bytes of each of 32. Piece c (16 bytes) of row r lies at
// piece c ^ (r % 8): neither the rows' pieces going in nor the rows coming out meet in a bank.
template <int DIM> struct StagedRows {
    static constexpr int PIECES = DIM / 8;
    static constexpr int ROWS_AT_ONCE = 32 / PIECES;
    uint32_t rows_base; // shared-memory address

    __device__ __forceinline__ uint32_t address(int row, int piece) const {
        return rows_base + (row * PIECES + (piece ^ (row % 8))) * 16;
    }
    __device__ __forceinline__ void put(int row, int piece, uint4 value) const {
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address(row, piece)),
                     "r"(value.x), "r"(value.y), "r"(value.z), "r"(value.w)
                     : "memory");
    }
    // The first `rows` rows, `stride` elements apart. The whole warp calls it.
    __device__ __forceinline__ void store(uint16_t *output, int64_t stride, int rows) const {
        const int lane = threadIdx.x % 32;
        const int piece = lane % PIECES;
        __syncwarp();
        #pragma unroll
        for (int pass = 0; pass < 32 / ROWS_AT_ONCE; pass++) {
            const int row = pass * ROWS_AT_ONCE + lane / PIECES;
            if (row < rows) {
                uint4 value;
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(value.x), "=r"(value.y), "=r"(value.z), "=r"(value.w)
                             : "r"(address(row, piece))
                             : "memory");
                *reinterpret_cast<uint4 *>(output + row * stride + piece * 8) = value;
            }
        }
    }
};

// The larger of two values, a NaN if one of them is.
__device__ __forceinline__ float max_or_nan(float first, float second) {
    float result;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(result) : "f"(first), "f"(second));
    return result;
}

__device__ __forceinline__ float exp2_approx(float value) {
    float result;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(result) : "f"(value));
    return result;
}

// 2^x for both halves of a pair on the FMA pipe instead of the MUFU: x is split into its nearest
// integer n (the low mantissa bits after adding 1.5 * 2^23) and a fraction f in [-0.5, 0.5], 2^f is
// a polynomial of degree six, fitted for the smallest relative error (2.0e-9) with a constant term
// of one, and n goes into the exponent field. The result is within 8.0e-8 of 2^x, closer than
// ex2.approx, which is within 1.45e-7 (both over 200 million values from -125 to 8); a degree less
// gives 1.67e-7. x must not be far above zero. At -127 and below the bits come to exactly zero, as
// the MUFU has it, so that a masked key weighs nothing; what lies between there and -126 goes
// towards zero among the denormals. A NaN gives zero too: the caller looks for those itself.
__device__ __forceinline__ float2 exp2_polynomial(float2 x) {
    constexpr float MAGIC = 12582912.0f;
    constexpr float COEFFICIENTS[7] = {1.0f,
                                       0.6931471824645996f,
                                       0.24022647738456726f,
                                       0.055503323674201965f,
                                       0.00961843691766262f,
                                       0.0013398875016719103f,
                                       0.00015353361959569156f};
    x.x = fmaxf(x.x, -127.0f);
    x.y = fmaxf(x.y, -127.0f);
    const float2 shifted = __fadd2_rn(x, make_float2(MAGIC, MAGIC));
    const float2 whole = __fadd2_rn(shifted, make_float2(-MAGIC, -MAGIC));
    const float2 fraction = __ffma2_rn(whole, make_float2(-1.0f, -1.0f), x);
    float2 power = make_float2(COEFFICIENTS[6], COEFFICIENTS[6]);
    #pragma unroll
    for (int degree = 5; degree >= 0; degree--) {
        power = __ffma2_rn(power, fraction,
                           make_float2(COEFFICIENTS[degree], COEFFICIENTS[degree]));
    }
    power.x = __int_as_float(__float_as_int(power.x) + (__float_as_int(shifted.x) << 23));
    power.y = __int_as_float(__float_as_int(power.y) + (__float_as_int(shifted.y) << 23));
    return power;
}

// The sine (x) and cosine (y) of an angle of at most ANGLE_LIMIT without a branch, so that a thread's
// several are under way together: Cody and Waite's reduction by n quarter turns, pi/2 in three
// floats, each step one FMA; polynomials fitted over [-pi/4, pi/4] for the smallest relative error
// (7.9e-9 and 1.6e-10 as their coefficients are rounded); the quadrant by n's low bits. At most 1.55
// units in the last place off over 20 million angles up to the limit; sincosf is allowed two.
constexpr float ANGLE_LIMIT = 48000.0f;
__device__ __forceinline__ float2 sine_and_cosine(float angle) {
    const float n = rintf(angle * 0.636619772f);
    float r = fmaf(n, -1.5707963705062866f, angle);
    r = fmaf(n, 4.371138828673793e-08f, r);
    r = fmaf(n, 1.7151245100058819e-15f, r);
    const float z = r * r;
    float sine = fmaf(z, -0.0001951398007804528f, 0.008332150988280773f);
    sine = fmaf(z, sine, -0.16666653752326965f);
    sine = fmaf(r * z, sine, r);
    float cosine = fmaf(z, 2.4431667043245398e-05f, -0.0013887303648516536f);
    cosine = fmaf(z, cosine, 0.04166664555668831f);
    cosine = fmaf(z, cosine, -0.5f);
    cosine = fmaf(z, cosine, 1.0f);
    const uint32_t quarter = static_cast<uint32_t>(static_cast<int>(n));
    const float2 turned = quarter & 1u ? make_float2(cosine, sine) : make_float2(sine, cosine);
    return make_float2(
        __uint_as_float(__float_as_uint(turned.x) ^ (quarter << 30 & 0x80000000u)),
        __uint_as_float(__float_as_uint(turned.y) ^ ((quarter + 1u) << 30 & 0x80000000u)));
}

__device__ __forceinline__ uint32_t pack_bf16(float low, float high) {
    uint32_t packed;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(high), "f"(low));
    return packed;
}

} // namespace sm100
