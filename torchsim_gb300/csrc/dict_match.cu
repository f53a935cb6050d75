// Dictionary matching on the 5th-generation tensor cores.
//
// The reference's DictionaryMatcher (estimators/_dictionary.py:52-420) scores
// every normalized measurement against every normalized atom by |<s, d>|
// through chunked FP32 matrix products (_grouped.py:212-240) and keeps the
// top k. Here one kernel does the product and the selection without ever
// writing the score matrix: queries (two rows per voxel) and atoms are fp16
// K-major tiles brought by TMA into shared memory (the queries once per sweep
// over the atoms where they fit, the atoms through a ring);
// `tcgen05.mma` (issued by one thread) accumulates a 128 x 256 tile in tensor
// memory, double-buffered so the epilogue of one atom tile overlaps the MMAs of
// the next; eight epilogue warps (two per TMEM lane quarter, each taking every
// other 32-column chunk) read the accumulator with `tcgen05.ld`. The two lanes
// holding a voxel's rows exchange one value per pair of atoms; each (warp,
// lane) keeps its best kScreen atoms of one (chunk parity, column parity)
// class, so a voxel keeps kCand = 32; the atoms are stored permuted so that
// neighbouring atoms land in different classes. A chunk of atoms whose best
// does not beat a lane's current last place costs no insertion work. A second kernel rescores
// those candidates exactly in FP32 against the complex signals and atoms and
// keeps the top k, so the fp16 screen decides only which few atoms are
// compared exactly.
//
// Rows of the query matrix: voxel v owns rows 2v and 2v+1. For real atoms
// (an SSFP fingerprint) they are (Re s_v, Im s_v) against the atom; for
// complex atoms (Re s, Im s) and (Im s, -Re s) against (Re d, Im d), whose
// products are the real and imaginary parts of <s, d>.
//
// Bound: the tensor pipe and its power (1.8 to 1.9 PFLOP/s). Measured, 16,384
// voxels x 65,536 atoms x 500 samples: 3.62 ms with one CTA per 128 rows in
// whole waves, 3.24 with row tiles in pairs, the last wave split and resident
// queries, 3.16 with the pair's two SMs on one product, 2.95 with the
// candidates inserted a lane's best at a time, 2.43 (1.78 PFLOP/s) with one
// commit for a contraction tile; 1,024 voxels 2.0 -> 0.22 ms by the split. The
// rescoring, bound by reading the candidates' atoms, 367 -> 219 us by reading
// one part of atoms on an axis and four candidates at a time.
//
// Waits on mbarriers are bounded: a wait that runs out sets the error word
// and the kernel winds down instead of hanging.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "tsg_internal.h"

namespace tsg {

namespace {

constexpr int BM = 128, BN = 256, BK = 64;  // of one CTA's query rows; of a pair's atoms
constexpr int kScreen = 8;           // per lane
constexpr int kHalves = 2;            // epilogue warps per TMEM lane quarter
constexpr int kClasses = 2 * kHalves;
constexpr int kCand = kClasses * kScreen;  // per voxel
constexpr int SMEM_A = BM * BK * 2;
constexpr int SMEM_B = BN / 2 * BK * 2;  // a CTA's half
// CTAs come in pairs (a cluster, cta_group::2): 256 query rows against 256
// atoms a tile, each CTA holding its 128 query rows, its half of the atom
// tile and the accumulator of its rows. One CTA alone reads 96 bytes of
// shared memory a cycle for its products while 64 or more are written, which
// is past the 128 the memory has; half the atom tile makes it 64 and 32.
constexpr int kPair = 2;
// Shared-memory slots: query tiles resident for a whole sweep over the atoms
// where the contraction has at most kResident tiles; atom tiles in a ring, a
// slot holding all parts of a contraction tile and, where they are not
// resident, its query tile. One wait and one commit then go with all the
// products of a contraction tile: each tcgen05.commit holds up the products
// after it, and with one for every part and query tile the pipe stayed 60%
// active whatever the ring's depth (16,384 voxels x 65,536 atoms x 500 samples
// 2.95 and 2.43 ms). At whole waves the gain is as large as the power cap lets
// it: 65,536 x 262,144 x 880 against one CTA per 128 rows 84 and 70 ms after a
// pause, 88 and 75 back to back, on the MRF dictionary under the benchmark's
// load 78 and 78 to 79.
constexpr int kResident = 8;
constexpr int kMaxA = 8, kMaxB = 10;
constexpr int kTileBytes = 224 * 1024;  // of both
constexpr int TMEM_COLS = 2 * BN;
constexpr int kEpilogueThreads = 128 * kHalves;
// warp 0 TMA, warp 1 MMA + TMEM, warps 2.. epilogue (each lane quarter twice:
// one warp per half of the accumulator's columns).
constexpr int kThreads = 64 + kEpilogueThreads;
constexpr long long kWaitLimit = 1LL << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool wait_parity(uint32_t bar, uint32_t parity) {
    for (long long i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The screen matrix stores atom i at row pos(i), which moves bit 1 of i to
// bit 5 and bits 2-5 down by one, within blocks of 64: consecutive atoms then
// alternate in column parity and in 32-column chunk parity, so they fall in
// four different candidate lists of the voxel (dictionaries put neighbouring
// atoms next to each other). This is the inverse: the atom at row `pos`.
__host__ __device__ __forceinline__ int stored_atom(int pos) {
    return (pos & 1) | (((pos >> 5) & 1) << 1) | (((pos >> 1) & 15) << 2) | (pos & ~63);
}

// The same place in the shared memory of the pair's first CTA.
__device__ __forceinline__ uint32_t first_cta(uint32_t addr) {
    uint32_t there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(there) : "r"(addr));
    return there;
}

__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Both CTAs of a pair (every thread of each arrives, whatever happened).
__device__ __forceinline__ void pair_sync() {
    asm volatile(
        "barrier.cluster.arrive.release;\n"
        "barrier.cluster.wait.acquire;\n" ::
            : "memory");
}

// Shared-memory matrix descriptor of a K-major 16-bit tile with 128-byte
// swizzle: 8-row groups 1024 bytes apart, rows of 128 bytes.
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= uint64_t((addr & 0x3FFFF) >> 4);
    d |= uint64_t(16 >> 4) << 16;
    d |= uint64_t(1024 >> 4) << 32;
    d |= uint64_t(1) << 46;
    d |= uint64_t(2) << 61;
    return d;
}

// kind::f16 instruction descriptor: FP32 accumulate, fp16 A and B (format
// 0), both K-major, M = 2 BM (the pair's rows), N = BN.
constexpr uint32_t kInstr = (1u << 4) | (uint32_t(BN >> 3) << 17) | (uint32_t(kPair * BM >> 4) << 24);

// The full and tempty barriers of the pair's first CTA serve both: it issues
// the products. The others are each CTA's own, reached by multicast commits.
struct ScreenShared {
    uint64_t a_full[kMaxA];
    uint64_t a_empty[kMaxA];
    uint64_t b_full[kMaxB];
    uint64_t b_empty[kMaxB];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint32_t tmem_base;
    int abort;
};

// How the (pair of query row tiles) x (atom tile) plane is shared among the
// CTA pairs: items 0 .. full-1 are row pairs with all their atom tiles; the
// last `split` row pairs are cut into `pieces` runs of `run` atom tiles each,
// items in order of the run first, so that CTAs working side by side read the
// same few atom tiles. Pair c takes items c, c + pairs, ... A piece's
// candidates go to its own list, merged before the rescoring: piece p's list of
// voxel v is list p list_step + v. With list_step the voxels of the split row
// pairs there is one list for every voxel and one more of theirs per further
// piece (65,536 atoms: 58,496 voxels have one split row pair, in 32 pieces; a
// list for every voxel and piece took 479 MB there, this takes 16).
struct ScreenWork {
    int n_tiles;  // atom tiles
    int full, split, pieces, run;
    int k_tiles;  // contraction tiles of one part
    int parts;    // atom matrices side by side along the contraction (hi, lo)
    int k_step;   // columns from one part to the next
    int na, nb;   // slots
    int slot;     // bytes of a ring slot in one CTA
    bool resident;
    int64_t list_step;
};

struct ScreenItem {
    int row_pair, piece, begin, end;
};

__host__ __device__ __forceinline__ int screen_items(const ScreenWork& w) {
    return w.full + w.split * w.pieces;
}

__device__ __forceinline__ ScreenItem screen_item(const ScreenWork& w, int i) {
    if (i < w.full) return {i, 0, 0, w.n_tiles};
    const int j = i - w.full, piece = j / w.split;
    const int begin = piece * w.run;
    return {w.full + j % w.split, piece, begin, min(begin + w.run, w.n_tiles)};
}

#define TSG_LD32(r, taddr)                                                                         \
    asm volatile(                                                                                  \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14," \
        "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"             \
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),      \
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),  \
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),            \
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),            \
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])             \
        : "r"(taddr))

__global__ void __cluster_dims__(kPair, 1, 1) __launch_bounds__(kThreads, 1)
    screen_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap amap,
                  const __grid_constant__ ScreenWork w, int64_t rows, int64_t atoms,
                  float* cand_score, int32_t* cand_index, int* error) {
    extern __shared__ uint8_t s_raw[];
    uint8_t* a_tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* b_tiles = a_tiles + w.na * SMEM_A;
    ScreenShared* sh = reinterpret_cast<ScreenShared*>(b_tiles + w.nb * w.slot);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int items = screen_items(w);
    const int rank = int(blockIdx.x) % kPair;
    const int first_item = int(blockIdx.x) / kPair, item_step = int(gridDim.x) / kPair;
    constexpr uint16_t kBoth = (1u << kPair) - 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < w.na; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh->a_full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh->a_empty[s])));
        }
        for (int s = 0; s < w.nb; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh->b_full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh->b_empty[s])));
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh->tfull[b])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&sh->tempty[b])),
                         "r"(kPair * kEpilogueThreads / 32));
        }
        sh->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&sh->tmem_base)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_sync();  // both CTAs' barriers are set up
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh->tmem_base;
    volatile int* abort = &sh->abort;
    auto give_up = [&](int stage) {
        *abort = 1;
        atomicExch(error, stage);
    };

    if (warp == 0) {
        if (lane == 0) {
            // TMA producer.
            // Both CTAs' bytes of a slot land on the first CTA's barrier,
            // which that CTA arms for the sum.
            auto arm = [&](uint64_t* bar, int bytes) {
                if (rank == 0)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                                 "r"(kPair * bytes)
                                 : "memory");
            };
            auto fetch = [&](const CUtensorMap& map, uint8_t* to, uint64_t* bar, int x, int y) {
                asm volatile(
                    "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global"
                    ".mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(to)),
                    "l"(reinterpret_cast<uint64_t>(&map)), "r"(x), "r"(y), "r"(first_cta(smem_u32(bar)))
                    : "memory");
            };
            int as = 0, bs = 0;
            uint32_t ap = 1, bp = 1;  // parity of the slots' release
            for (int i = first_item; i < items && !*abort; i += item_step) {
                const ScreenItem it = screen_item(w, i);
                for (int n = it.begin; n < it.end && !*abort; ++n) {
                    for (int kt = 0; kt < w.k_tiles; ++kt) {
                        const int row = (it.row_pair * kPair + rank) * BM;
                        if (w.resident && n == it.begin) {
                            if (!wait_parity(smem_u32(&sh->a_empty[as]), ap)) {
                                give_up(1);
                                break;
                            }
                            arm(&sh->a_full[as], SMEM_A);
                            fetch(qmap, a_tiles + as * SMEM_A, &sh->a_full[as], kt * BK, row);
                            if (++as == w.na) {
                                as = 0;
                                ap ^= 1;
                            }
                        }
                        if (!wait_parity(smem_u32(&sh->b_empty[bs]), bp)) {
                            give_up(1);
                            break;
                        }
                        arm(&sh->b_full[bs], w.slot);
                        uint8_t* to = b_tiles + bs * w.slot;
                        if (!w.resident) {
                            fetch(qmap, to, &sh->b_full[bs], kt * BK, row);
                            to += SMEM_A;
                        }
                        for (int part = 0; part < w.parts; ++part)
                            fetch(amap, to + part * SMEM_B, &sh->b_full[bs],
                                  part * w.k_step + kt * BK, n * BN + rank * (BN / kPair));
                        if (++bs == w.nb) {
                            bs = 0;
                            bp ^= 1;
                        }
                    }
                }
            }
            // Every release of a slot, sent by the first CTA, has arrived
            // before this CTA can end.
            for (int j = 0; j < w.nb && !*abort; ++j) {
                if (!wait_parity(smem_u32(&sh->b_empty[bs]), bp)) give_up(1);
                if (++bs == w.nb) {
                    bs = 0;
                    bp ^= 1;
                }
            }
            for (int j = 0; j < w.na && !*abort; ++j) {
                if (!wait_parity(smem_u32(&sh->a_empty[as]), ap)) give_up(1);
                if (++as == w.na) {
                    as = 0;
                    ap ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // MMA issuer, for the pair. A commit arrives on both CTAs' barrier.
            auto commit = [&](uint64_t* bar) {
                asm volatile(
                    "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster"
                    ".multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                    "h"(kBoth)
                    : "memory");
            };
            int bs = 0;
            uint32_t ap = 0, bp = 0;
            int t = 0;  // tiles so far: the accumulator is t & 1
            for (int i = first_item; i < items && !*abort; i += item_step) {
                const ScreenItem it = screen_item(w, i);
                for (int n = it.begin; n < it.end && !*abort; ++n, ++t) {
                    const int b = t & 1;
                    if (!wait_parity(smem_u32(&sh->tempty[b]), ((t >> 1) & 1) ^ 1)) {
                        give_up(2);
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + uint32_t(b * BN);
                    uint32_t acc = 0;
                    for (int kt = 0; kt < w.k_tiles; ++kt) {
                        if (w.resident && n == it.begin &&
                            !wait_parity(smem_u32(&sh->a_full[kt]), ap)) {
                            give_up(3);
                            break;
                        }
                        if (!wait_parity(smem_u32(&sh->b_full[bs]), bp)) {
                            give_up(3);
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        uint32_t b_addr = smem_u32(b_tiles + bs * w.slot);
                        uint32_t a_addr = b_addr;
                        if (w.resident)
                            a_addr = smem_u32(a_tiles + kt * SMEM_A);
                        else
                            b_addr += SMEM_A;
                        for (int part = 0; part < w.parts; ++part, b_addr += SMEM_B) {
#pragma unroll
                            for (int j = 0; j < BK / 16; ++j) {
                                const uint64_t adesc = tile_desc(a_addr + j * 32);
                                const uint64_t bdesc = tile_desc(b_addr + j * 32);
                                asm volatile(
                                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                                    "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
                                    "l"(adesc), "l"(bdesc), "r"(kInstr), "r"(acc)
                                    : "memory");
                                acc = 1;
                            }
                        }
                        commit(&sh->b_empty[bs]);
                        if (++bs == w.nb) {
                            bs = 0;
                            bp ^= 1;
                        }
                        if (w.resident && n + 1 == it.end) commit(&sh->a_empty[kt]);
                    }
                    if (*abort) break;
                    commit(&sh->tfull[b]);
                }
                ap ^= 1;
            }
        }
    } else {
        // Epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 = tile rows, in
        // the columns of its half of the accumulator. A voxel's rows sit on
        // lanes 2i (Re) and 2i+1 (Im); lane parity p scores the atoms of
        // column parity p.
        const int quarter = warp & 3;
        const int half = (warp - 2) / 4;
        const int r = quarter * 32 + lane;
        const int parity = lane & 1;
        const int64_t whole = atoms & ~int64_t(63);  // rows below hold atoms only
        int t = 0;
        for (int i = first_item; i < items && !*abort; i += item_step) {
            const ScreenItem it = screen_item(w, i);
            float best_s[kScreen];
            int best_i[kScreen];
#pragma unroll
            for (int k = 0; k < kScreen; ++k) {
                best_s[k] = -1.f;
                best_i[k] = -1;
            }
            for (int n = it.begin; n < it.end && !*abort; ++n, ++t) {
                const int b = t & 1;
                if (!wait_parity(smem_u32(&sh->tfull[b]), (t >> 1) & 1)) {
                    give_up(4);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int cc = 0; cc < BN / 64; ++cc) {
                    // The warp of half h takes the 32-column chunks of parity h.
                    const int c = 2 * cc + half;
                    uint32_t v[32];
                    const uint32_t taddr = tmem + (uint32_t(quarter * 32) << 16) + uint32_t(b * BN + c * 32);
                    TSG_LD32(v, taddr);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float sc[16];
                    float chunk_best = -1.f;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float x0 = __uint_as_float(v[2 * j]), x1 = __uint_as_float(v[2 * j + 1]);
                        // Send the partner the value of its column; keep our own.
                        const float mine = parity ? x1 : x0;
                        const float other = __shfl_xor_sync(0xffffffffu, parity ? x0 : x1, 1);
                        sc[j] = fmaf(mine, mine, other * other);
                        chunk_best = fmaxf(chunk_best, sc[j]);
                    }
                    const int pos0 = n * BN + c * 32 + parity;
                    if (n * BN + c * 32 + 32 > whole) {
                        // The last atoms' block: rows past the end do not count.
                        chunk_best = -1.f;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (stored_atom(pos0 + 2 * j) >= atoms) sc[j] = -1.f;
                            chunk_best = fmaxf(chunk_best, sc[j]);
                        }
                    }
                    // Each round takes every lane's best remaining score at
                    // once, so the warp pays for the lane with the most.
                    while (__any_sync(0xffffffffu, chunk_best > best_s[kScreen - 1])) {
                        const float score = chunk_best;
                        const bool take = score > best_s[kScreen - 1];
                        int at = 0;
                        float rest = -1.f;
#pragma unroll
                        for (int j = 15; j >= 0; --j) {
                            if (sc[j] == score) at = j;
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            if (j == at) sc[j] = -1.f;
                            rest = fmaxf(rest, sc[j]);
                        }
                        chunk_best = rest;
                        const int atom = stored_atom(pos0 + 2 * at);
                        best_s[kScreen - 1] = take ? score : best_s[kScreen - 1];
                        best_i[kScreen - 1] = take ? atom : best_i[kScreen - 1];
#pragma unroll
                        for (int k = kScreen - 1; k > 0; --k) {
                            const bool up = best_s[k] > best_s[k - 1];
                            const float hi = up ? best_s[k] : best_s[k - 1];
                            const float lo = up ? best_s[k - 1] : best_s[k];
                            const int hi_i = up ? best_i[k] : best_i[k - 1];
                            const int lo_i = up ? best_i[k - 1] : best_i[k];
                            best_s[k - 1] = hi;
                            best_s[k] = lo;
                            best_i[k - 1] = hi_i;
                            best_i[k] = lo_i;
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive_cluster(first_cta(smem_u32(&sh->tempty[b])));
            }
            const int64_t row = int64_t(it.row_pair * kPair + rank) * BM + (r & ~1);
            if (row < rows && !*abort) {
                const int64_t at = (int64_t(it.piece) * w.list_step + (row >> 1)) * kCand +
                                   (half * 2 + parity) * kScreen;
#pragma unroll
                for (int k = 0; k < kScreen; ++k) {
                    cand_score[at + k] = best_s[k];
                    cand_index[at + k] = best_i[k];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort) {
        // Let copies and products in flight land before the memory goes away.
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    // The other CTA may still copy into this one's slots and arrive on its
    // barriers until it is done too.
    pair_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(TMEM_COLS));
}

// Two fp16 rows per normalized signal (see the head of this file), scaled,
// zero-padded to `k` columns. One warp per voxel.
__global__ void query_kernel(const float2* __restrict__ signals, int64_t voxels, int64_t samples,
                             int64_t k, float scale, bool complex_atoms, __half* __restrict__ out) {
    const int64_t voxel = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (voxel >= voxels) return;
    const float2* s = signals + voxel * samples;
    __half* a = out + 2 * voxel * k;
    __half* b = a + k;
    for (int64_t p = lane; p < k; p += 32) {
        float x = 0.f, y = 0.f;
        if (p < samples) {
            const float2 v = s[p];
            x = v.x;
            y = v.y;
        } else if (complex_atoms && p < 2 * samples) {
            const float2 v = s[p - samples];
            x = v.y;
            y = -v.x;
        }
        a[p] = __float2half_rn(x * scale);
        b[p] = __float2half_rn(y * scale);
    }
}

// Keeps in (s, x) the best kScreen of two lists sorted best first, ties to the
// first: the larger of opposite ends is the set, as a bitonic sequence.
__device__ __forceinline__ void merge_lists(float (&s)[kScreen], int (&x)[kScreen],
                                            const float (&t)[kScreen], const int (&y)[kScreen]) {
#pragma unroll
    for (int k = 0; k < kScreen; ++k) {
        const bool other = t[kScreen - 1 - k] > s[k];
        s[k] = other ? t[kScreen - 1 - k] : s[k];
        x[k] = other ? y[kScreen - 1 - k] : x[k];
    }
#pragma unroll
    for (int half = kScreen / 2; half > 0; half >>= 1)
#pragma unroll
        for (int k = 0; k < kScreen; ++k) {
            if (k & half) continue;
            const bool swap = s[k + half] > s[k];
            const float hi = swap ? s[k + half] : s[k], lo = swap ? s[k] : s[k + half];
            const int hx = swap ? x[k + half] : x[k], lx = swap ? x[k] : x[k + half];
            s[k] = hi;
            s[k + half] = lo;
            x[k] = hx;
            x[k + half] = lx;
        }
}

// The merged candidate of this lane (class lane / kScreen, rank lane %
// kScreen) of `count` lists of the same voxel, `step` entries apart: per class
// the best kScreen of the lists' (each sorted best first) -- what one list
// over all the atoms would hold. A class's eight lanes look after every eighth
// list each and hand out the best of their heads in turn.
__device__ __forceinline__ int merged_candidate(const float* score, const int32_t* index, int64_t at,
                                                int64_t step, int count, int lane) {
    static_assert(kClasses * kScreen == 32 && kScreen == 8, "a lane per candidate");
    if (count == 1) return index[at + lane];
    const int g = lane & 7;
    const int64_t mine0 = at + (lane & ~7);
    float s[kScreen];
    int x[kScreen];
    auto read = [&](int list, float (&u)[kScreen], int (&v)[kScreen]) {
#pragma unroll
        for (int k = 0; k < kScreen; ++k) {
            u[k] = list < count ? score[mine0 + list * step + k] : -2.f;
            v[k] = list < count ? index[mine0 + list * step + k] : -1;
        }
    };
    read(g, s, x);
    for (int list = g + 8; list - g < count; list += 8) {
        float t[kScreen];
        int y[kScreen];
        read(list, t, y);
        merge_lists(s, x, t, y);
    }
    int mine = -1;
#pragma unroll
    for (int k = 0; k < kScreen; ++k) {
        float best = s[0];
        int from = g;
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, best, off);
            const int f = __shfl_xor_sync(0xffffffffu, from, off);
            if (o > best || (o == best && f < from)) {
                best = o;
                from = f;
            }
        }
        const int atom = __shfl_sync(0xffffffffu, x[0], (lane & ~7) + from);
        if (g == k) mine = atom;
        const bool mine_won = g == from;
#pragma unroll
        for (int j = 0; j + 1 < kScreen; ++j) {
            s[j] = mine_won ? s[j + 1] : s[j];
            x[j] = mine_won ? x[j + 1] : x[j];
        }
        if (mine_won) {
            s[kScreen - 1] = -2.f;
            x[kScreen - 1] = -1;
        }
    }
    return mine;
}

// Exact FP32 rescoring of each voxel's screened candidates against the complex
// normalized signal and atoms; keeps the best `top_k` in descending order.
// One warp per voxel: lanes stride over the samples. Bound by reading the
// candidates' atoms, so a dictionary on one axis is read as its one part:
// AXIS 0 complex atoms, 1 real, 2 on the imaginary axis (the products with
// the other part, zero, leave the sums as they are).
template <int AXIS>
__global__ void rescore_kernel(const float2* __restrict__ signals, const void* __restrict__ atoms,
                               int64_t voxels, int64_t samples, const float* __restrict__ list_score,
                               const int32_t* __restrict__ list_index, int full_pairs, int pieces,
                               int64_t list_step, int top_k, float* __restrict__ scores, int64_t* __restrict__ index) {
    const int64_t voxel = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (voxel >= voxels) return;
    const int count = 2 * voxel / (BM * kPair) < full_pairs ? 1 : pieces;
    int mine = merged_candidate(list_score, list_index, voxel * kCand, list_step * kCand, count, lane);
    const float2* s = signals + voxel * samples;
    float my_score = -1.f;
    // Four candidates at a time, whose loads overlap and share the signal's.
    constexpr int kTogether = 4;
#pragma unroll 1
    for (int k = 0; k < kCand; k += kTogether) {
        int atom[kTogether];
        float re[kTogether], im[kTogether];
        const void* row[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
            atom[j] = __shfl_sync(0xffffffffu, mine, k + j);
            re[j] = im[j] = 0.f;
            const int64_t at = int64_t(max(atom[j], 0)) * samples;
            row[j] = AXIS == 0 ? static_cast<const void*>(static_cast<const float2*>(atoms) + at)
                               : static_cast<const void*>(static_cast<const float*>(atoms) + at);
        }
#pragma unroll 2
        for (int64_t p = lane; p < samples; p += 32) {
            const float2 x = s[p];
#pragma unroll
            for (int j = 0; j < kTogether; ++j) {
                if constexpr (AXIS == 0) {
                    const float2 y = static_cast<const float2*>(row[j])[p];
                    // s * conj(d)
                    re[j] = fmaf(x.x, y.x, fmaf(x.y, y.y, re[j]));
                    im[j] = fmaf(x.y, y.x, fmaf(-x.x, y.y, im[j]));
                } else {
                    const float y = static_cast<const float*>(row[j])[p];
                    if constexpr (AXIS == 1) {
                        re[j] = fmaf(x.x, y, re[j]);
                        im[j] = fmaf(x.y, y, im[j]);
                    } else {
                        re[j] = fmaf(x.y, y, re[j]);
                        im[j] = fmaf(-x.x, y, im[j]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                re[j] += __shfl_xor_sync(0xffffffffu, re[j], off);
                im[j] += __shfl_xor_sync(0xffffffffu, im[j], off);
            }
            if (lane == k + j && atom[j] >= 0) my_score = sqrtf(re[j] * re[j] + im[j] * im[j]);
        }
    }
    // Descending by score, ties to the lower atom index; -1 where none is left.
    for (int k = 0; k < top_k; ++k) {
        float best = my_score;
        int atom = mine;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, best, off);
            const int a = __shfl_xor_sync(0xffffffffu, atom, off);
            if (o > best || (o == best && a >= 0 && (atom < 0 || a < atom))) {
                best = o;
                atom = a;
            }
        }
        if (lane == 0) {
            scores[voxel * top_k + k] = best;
            index[voxel * top_k + k] = atom;
        }
        if (mine == atom) {
            my_score = -1.f;
            mine = -1;
        }
    }
}

// What goes with the atoms found: the least-squares scale <d, s> / |d|^2 of
// the signals as given, its size from the score, and the atoms' parameters.
// One warp per voxel and place.
__global__ void result_kernel(const float2* __restrict__ signals, const float* __restrict__ norms,
                              int64_t found, int64_t samples, int top_k, int64_t atoms,
                              const float2* __restrict__ dictionary, const float* __restrict__ power,
                              const float* __restrict__ scores, const int64_t* __restrict__ index,
                              const float* __restrict__ table, int columns,
                              float2* __restrict__ scales, float* __restrict__ densities,
                              float* __restrict__ parameters) {
    const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= found) return;
    const int64_t voxel = i / top_k;
    // A signal that matches nothing (a NaN in it) has index -1, which reads as
    // the last atom, as indexing from the end does.
    const int64_t atom = index[i] < 0 ? atoms - 1 : index[i];
    const float2* s = signals + voxel * samples;
    const float2* d = dictionary + atom * samples;
    float re = 0.f, im = 0.f;
    for (int64_t p = lane; p < samples; p += 32) {
        const float2 x = s[p], y = d[p];
        re = fmaf(x.x, y.x, fmaf(x.y, y.y, re));
        im = fmaf(x.y, y.x, fmaf(-x.x, y.y, im));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, off);
        im += __shfl_xor_sync(0xffffffffu, im, off);
    }
    for (int c = lane; c < columns; c += 32) parameters[i * columns + c] = table[atom * columns + c];
    if (lane == 0) {
        const float pw = power[atom];
        scales[i] = make_float2(re / pw, im / pw);
        densities[i] = norms[voxel] * scores[i] / sqrtf(pw);
    }
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return EncodeTiled(nullptr);
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

int tile_map(CUtensorMap* map, const void* base, int64_t rows, int64_t k, int box_rows) {
    EncodeTiled fn = encode_fn();
    if (!fn) return fail(TSG_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(k) * 2};
    const cuuint32_t box[2] = {cuuint32_t(BK), cuuint32_t(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims,
                          strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TSG_ERR_ARGUMENT, "tensor map rejected the matrix");
    return TSG_OK;
}

}  // namespace

}  // namespace tsg

using namespace tsg;

extern "C" int tsg_match_screen_rows(int64_t atom_count) {
    return int((atom_count + 63) / 64 * 64);
}

namespace tsg {
namespace {

int match_sms() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// The work split over the CTA pairs of `sms` SMs. Row pairs that fill whole
// waves stay whole; the rest are cut so that the last waves are full: the number of
// pieces that minimises waves x (piece + 2 tiles of filling and draining the
// pipeline), up to 32 lists a voxel and at least 8 tiles a piece. At 16,384
// voxels x 65,536 atoms (256 row tiles, 256 atom tiles, 152 SMs) two waves of
// 256 tiles become 256 + 3 x 64; at 1,024 voxels one wave of 256 becomes 29.
ScreenWork plan_screen(int64_t query_rows, int64_t atom_count, int64_t k, int parts, int sms,
                       bool may_split) {
    ScreenWork w{};
    const int pairs = int((query_rows + kPair * BM - 1) / (kPair * BM));
    const int slots = std::max(1, sms / kPair);
    const int64_t stored = (atom_count + 63) / 64 * 64;
    w.n_tiles = int((stored + BN - 1) / BN);
    w.parts = parts;
    w.k_step = int(k);
    w.k_tiles = int((k + BK - 1) / BK);
    w.resident = w.k_tiles <= kResident;
    w.na = w.resident ? w.k_tiles : 0;
    w.slot = w.parts * SMEM_B + (w.resident ? 0 : SMEM_A);
    w.nb = std::min(kMaxB, (kTileBytes - w.na * SMEM_A) / w.slot);
    w.full = may_split ? pairs / slots * slots : pairs;
    w.split = pairs - w.full;
    w.list_step = std::max<int64_t>(0, query_rows / 2 - int64_t(w.full) * (kPair * BM / 2));
    w.pieces = 1;
    w.run = w.n_tiles;
    double best = 1e300;
    for (int p = 1; w.split > 0 && p <= 32 && (p == 1 || w.n_tiles / p >= 8); ++p) {
        const int run = (w.n_tiles + p - 1) / p;
        const int pieces = (w.n_tiles + run - 1) / run;  // none empty
        const int64_t waves = (int64_t(w.split) * pieces + slots - 1) / slots;
        const double cost = double(waves) * (run + 2);
        if (cost < best) {
            best = cost;
            w.run = run;
            w.pieces = pieces;
        }
    }
    return w;
}

int check_screen(const void* queries, int64_t query_rows, const void* atoms, int64_t atom_count,
                 int64_t k, const void* scores, const void* index, const void* error) {
    if (query_rows < 0 || atom_count < 0 || k < 1)
        return fail(TSG_ERR_ARGUMENT, "invalid matching dimensions");
    if (query_rows % 2) return fail(TSG_ERR_ARGUMENT, "queries come as two rows per voxel");
    if (k % 8) return fail(TSG_ERR_ARGUMENT, "the inner dimension must be a multiple of 8 (16 bytes)");
    if (query_rows == 0) return TSG_OK;
    if (!queries || !atoms || !scores || !index || !error)
        return fail(TSG_ERR_ARGUMENT, "null matching buffer");
    if ((reinterpret_cast<uintptr_t>(queries) | reinterpret_cast<uintptr_t>(atoms)) & 15)
        return fail(TSG_ERR_ARGUMENT, "matrices must be 16-byte aligned");
    if (atom_count == 0) return fail(TSG_ERR_ARGUMENT, "empty dictionary");
    if (query_rows > (int64_t(1) << 31) - BM || atom_count > (int64_t(1) << 31) - BN ||
        k > (int64_t(1) << 29))
        return fail(TSG_ERR_CAPACITY, "matrix too large");
    return TSG_OK;
}

int run_screen(const ScreenWork& w, const void* queries, int64_t query_rows, const void* atoms,
               int64_t atom_count, int64_t k, float* scores, int32_t* index, int* error, int sms,
               cudaStream_t stream) {
    CUtensorMap qmap, amap;
    const int64_t stored_rows = (atom_count + 63) / 64 * 64;
    int rc = tile_map(&qmap, queries, query_rows, k, BM);
    if (!rc) rc = tile_map(&amap, atoms, stored_rows, k * w.parts, BN / kPair);
    if (rc) return rc;
    const size_t smem = 1024 + w.na * SMEM_A + w.nb * w.slot + sizeof(ScreenShared);
    TSG_CUDA(cudaFuncSetAttribute(screen_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    const int grid = kPair * std::min(std::max(1, sms / kPair), screen_items(w));
    screen_kernel<<<unsigned(grid), kThreads, smem, stream>>>(
        qmap, amap, w, query_rows, atom_count, scores, index, error);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

template <int AXIS>
void run_rescore(const void* signals, int64_t voxels, const void* atoms, int64_t samples,
                 const float* list_score, const int32_t* list_index, int full_pairs, int pieces,
                 int64_t list_step, int top_k, float* scores, int64_t* index, cudaStream_t stream) {
    rescore_kernel<AXIS><<<unsigned((voxels * 32 + 255) / 256), 256, 0, stream>>>(
        static_cast<const float2*>(signals), atoms, voxels, samples, list_score, list_index,
        full_pairs, pieces, list_step, top_k, scores, index);
}

}  // namespace
}  // namespace tsg

extern "C" int tsg_match_screen(const void* queries, int64_t query_rows, const void* atoms,
                                int64_t atom_count, int64_t k, float* candidate_scores,
                                int32_t* candidate_index, int* error, void* stream) {
    const int rc = check_screen(queries, query_rows, atoms, atom_count, k, candidate_scores,
                                candidate_index, error);
    if (rc || query_rows == 0) return rc;
    const int sms = match_sms();
    return run_screen(plan_screen(query_rows, atom_count, k, 1, sms, false), queries, query_rows, atoms,
                      atom_count, k, candidate_scores, candidate_index, error, sms,
                      static_cast<cudaStream_t>(stream));
}

extern "C" int tsg_match_rescore(const void* signals, int64_t voxels, const void* atoms,
                                 int64_t atom_count, int64_t samples,
                                 const int32_t* candidate_index, int top_k, float* scores,
                                 int64_t* index, void* stream) {
    if (voxels < 0 || atom_count < 1 || samples < 1 || top_k < 1 || top_k > 8)
        return fail(TSG_ERR_ARGUMENT, "invalid rescoring dimensions (top_k must be 1..8)");
    if (voxels == 0) return TSG_OK;
    if (!signals || !atoms || !candidate_index || !scores || !index)
        return fail(TSG_ERR_ARGUMENT, "null rescoring buffer");
    run_rescore<0>(signals, voxels, atoms, samples, nullptr, candidate_index, 0, 1, 0, top_k, scores,
                   index, static_cast<cudaStream_t>(stream));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_match_queries(const void* normalized, int64_t voxels, int64_t samples, int64_t k,
                                 float scale, int complex_atoms, void* queries, void* stream) {
    if (voxels < 0 || samples < 1 || k < (complex_atoms ? 2 : 1) * samples)
        return fail(TSG_ERR_ARGUMENT, "invalid query dimensions");
    if (voxels == 0) return TSG_OK;
    if (!normalized || !queries) return fail(TSG_ERR_ARGUMENT, "null matching buffer");
    query_kernel<<<unsigned((voxels * 32 + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(normalized), voxels, samples, k, scale, complex_atoms != 0,
        static_cast<__half*>(queries));
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_match_screen_lists(const void* queries, int64_t query_rows, const void* atoms,
                                      int64_t atom_count, int64_t k, float* list_scores,
                                      int32_t* list_index, int* error, void* stream) {
    const int rc = check_screen(queries, query_rows, atoms, atom_count, k, list_scores, list_index,
                                error);
    if (rc || query_rows == 0) return rc;
    const int sms = match_sms();
    ScreenWork w = plan_screen(query_rows, atom_count, k, 2, sms, true);
    w.list_step = query_rows / 2;
    return run_screen(w, queries, query_rows, atoms, atom_count, k, list_scores, list_index, error, sms,
                      static_cast<cudaStream_t>(stream));
}

extern "C" int tsg_match_lists(int64_t voxels, int64_t atom_count, int64_t k) {
    if (voxels < 1 || atom_count < 1 || k < 1) return 1;
    return plan_screen(2 * voxels, atom_count, k, 2, match_sms(), true).pieces;
}

extern "C" int64_t tsg_match_list_rows(int64_t voxels, int64_t atom_count, int64_t k) {
    if (voxels < 1 || atom_count < 1 || k < 1) return 1;
    const ScreenWork w = plan_screen(2 * voxels, atom_count, k, 2, match_sms(), true);
    return voxels + (w.pieces - 1) * w.list_step;
}

extern "C" int tsg_match(const tsg_match_dictionary* d, const void* signals, const void* normalized,
                         const float* norms, int64_t voxels, int top_k, void* queries,
                         float* list_scores, int32_t* list_index, int* error, float* scores,
                         int64_t* index, void* scales, float* densities, float* parameters,
                         void* stream) {
    if (!d || voxels < 0 || top_k < 1 || top_k > 8)
        return fail(TSG_ERR_ARGUMENT, "invalid matching dimensions (top_k must be 1..8)");
    if (d->samples < 1 || d->axis < 0 || d->axis > 2)
        return fail(TSG_ERR_ARGUMENT, "invalid matching dictionary");
    const int64_t need = d->axis == 0 ? 2 * d->samples : d->samples;
    if (d->k < need) return fail(TSG_ERR_ARGUMENT, "the contraction is shorter than the signals");
    const int rc = check_screen(queries, 2 * voxels, d->screen_atoms, d->atom_count, d->k, list_scores,
                                list_index, error);
    if (rc || voxels == 0) return rc;
    if (!signals || !normalized || !norms || !scores || !index || !scales || !densities ||
        !d->normalized_atoms || !d->dictionary || !d->power || (d->columns > 0 && (!d->table || !parameters)))
        return fail(TSG_ERR_ARGUMENT, "null matching buffer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int sms = match_sms();
    const ScreenWork w = plan_screen(2 * voxels, d->atom_count, d->k, 2, sms, true);
    int run = tsg_match_queries(normalized, voxels, d->samples, d->k, d->scale, d->axis == 0, queries, stream);
    if (!run)
        run = run_screen(w, queries, 2 * voxels, d->screen_atoms, d->atom_count, d->k, list_scores,
                         list_index, error, sms, s);
    if (run) return run;
    auto rescore = d->axis == 0 ? &run_rescore<0> : (d->axis == 1 ? &run_rescore<1> : &run_rescore<2>);
    rescore(normalized, voxels, d->normalized_atoms, d->samples, list_scores, list_index, w.full,
            w.pieces, w.list_step, top_k, scores, index, s);
    TSG_CUDA(cudaGetLastError());
    const int64_t found = voxels * top_k;
    result_kernel<<<unsigned((found * 32 + 255) / 256), 256, 0, s>>>(
        static_cast<const float2*>(signals), norms, found, d->samples, top_k, d->atom_count,
        static_cast<const float2*>(d->dictionary), d->power, scores, index, d->table,
        int(d->columns), static_cast<float2*>(scales), densities, parameters);
    TSG_CUDA(cudaGetLastError());
    return TSG_OK;
}

extern "C" int tsg_match_candidates(void) { return kCand; }
