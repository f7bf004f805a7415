// spx_launch.cuh -- launch sequences for one hash family instantiation.
//
// Each translation unit (spx_family_*.cu) instantiates Family<HF> for its
// (hash, n, robust) combinations and registers them in the dispatch table
// that the host engine indexes by parameter set.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "spx_kernels.cuh"
#include "spx_verify.cuh"
#include "spx_vblock.cuh"
#include "spx_vsort.cuh"

namespace cuspx {

// launch mapping knobs (picked per parameter set by the autotuner)
struct Tuning {
    int leaf_block = 128;    // threads per block for k_leaves
    int fors_block = 128;    // threads per block for k_fors_sign (multiple of 32)
    int verify_block = 64;   // threads per block for k_verify_root (and k_verify_ht)
    int tree_warps = 4;      // warps per block for k_trees (upper bound)
    int chains_per_warp = 64;  // (item, chain) tasks per warp in k_verify_chains
    int verify_mode = 0;     // 0 layered kernels, 1 one thread per item over all layers,
                             // 2 one launch over the hypertree, 3 layered with sorted chains
    int fors_lanes_log2 = 5; // lanes per FORS tree = 2^g (0: lane per tree, 5: warp per tree)
    int tree_mode = 0;       // 0 warp per XMSS tree, 1 lane per tree (subtrees of height <= 4)
    int chain_mode_max = 64; // sign batches of at most this many items take the T_len kernel of the
                             // lower latency; 0: XMSS leaves a lane each (up to kChainModeItems, and
                             // key generation)
    int verify_slots = 4;    // most items per warp in the persistent verify kernel (SHAKE)
    int verify_item_max = 0; // batches of at most this many items verify in one launch
    int verify_claim_min = 1;// persistent verify: free lanes before chains are handed out
    int verify_groups = 4;   // sorted verify: item groups on their own streams (1..8)
    int verify_sorted_min = 0; // batches of at least this many items verify as verify_mode 3 (0: never by size)
    int verify_spec_max = 0;   // batches of at most this many items verify with speculative chains (0: never)
};

struct KeygenArgs {
    uint32_t count;
    uint8_t *sk;       // count x 4n: SK_SEED || SK_PRF || PUB_SEED filled in, ROOT written
    uint8_t *pk;       // count x 2n: written
    uint8_t *leaves;   // count x 2^hp x n scratch
    uint8_t *roots;    // count x n scratch
    uint8_t *ends;        // chain-parallel scratch (ends_trees x 2^hp x len x n) or null
    uint32_t ends_trees;
    uint32_t *mids;       // SHA-256: 8 words per key
};

// Optional per-kernel timing: an event is recorded on the launch stream
// after every kernel of a sequence (event 0 before the first).
struct PhaseTimer {
    static constexpr int kMax = 160;
    cudaEvent_t ev[kMax + 1];
    const char *names[kMax];
    int n = 0;
    void mark(const char *name, cudaStream_t s) {
        if (n < kMax) {
            names[n] = name;
            cudaEventRecord(ev[n + 1], s);
            n++;
        }
    }
};
#define CUSPX_MARK(pt, name, s) \
    do {                        \
        if (pt) (pt)->mark(name, s); \
    } while (0)

// A side stream for the part of a sign sequence that runs beside the rest:
// the FORS trees need only the message digest, and the hypertree leaves and
// trees do not need FORS, so k_fors_sign runs on `side` between `fork`
// (recorded after the message kernels) and `join` (waited before
// k_sign_finish).  Works inside graph capture as a fork/join of the graph.
struct StreamFork {
    cudaStream_t side;
    cudaEvent_t fork, join;
};

// Streams of a verify batch for verify_mode 3: group g > 0 runs on side[g-1]
// between `fork` and join[g-1]; chain[g] orders group g+1's chain kernel of a
// layer after group g's.  Works inside graph capture.
struct VerifyFork {
    static constexpr int kMaxGroups = 8;
    int sides = 0;   // side streams available (groups beyond sides + 1 are not used)
    cudaStream_t side[kMaxGroups - 1] = {};
    cudaEvent_t fork = nullptr, join[kMaxGroups - 1] = {}, chain[kMaxGroups - 1] = {};
};

struct FamilyOps {
    cudaError_t (*configure)();
    // long_msg: messages of at least this many bytes are hashed two warps per
    // 32 messages (SHA-256) or a warp each (SHAKE-256); 0: none.
    // fk: optional side stream (ignored while per-kernel timing is on).
    void (*sign)(const SetParams &, SignArgs, const Tuning &, cudaStream_t, PhaseTimer *, uint64_t long_msg,
                 const StreamFork *fk);
    // vl / vf: bucket lists and streams of verify_mode 3 (null: that mode
    // runs as verify_mode 2)
    void (*verify)(const SetParams &, const VerifyArgs &, const Tuning &, cudaStream_t, PhaseTimer *,
                   uint64_t long_msg, const VerifyLists *vl, const VerifyFork *vf);
    void (*keygen)(const SetParams &, const KeygenArgs &, const Tuning &, cudaStream_t, PhaseTimer *);
    int smem_words;    // per-thread T_l stream scratch
};

// registry: [hash][n index 0..2][robust]
extern FamilyOps g_family[2][3][2];

// Shared trees of a sign batch (ShareArgs): the first layer with at most 8
// trees per item, and the entries of one layer's table.
inline int shared_layer0(const SetParams &P, uint64_t count) {
    int L = P.d - 1;
    while (L > 1 && (P.d - L) * P.hp < 40 && (1ull << ((P.d - L) * P.hp)) <= 8 * count) L--;
    return L;
}
inline uint32_t share_table(uint64_t count) {
    uint32_t n = 64;
    while (n < 2 * count) n *= 2;
    return n;
}

// Sign batches that chain_mode_max decides about.  Larger ones always run a
// lane per WOTS+ chain and look for shared trees (1024 signatures of 128f:
// 5.38 ms, a lane per leaf 5.99).
constexpr uint32_t kChainModeItems = 256;

inline unsigned ceil_div(uint64_t a, uint64_t b) { return (unsigned)((a + b - 1) / b); }

// SM count of the current device, queried once per device (a launch-shape
// input of the small-batch mappings; 1 if the query fails)
inline int device_sms() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v <= 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        v = sms > 0 ? sms : 1;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

// SHA-256 batches whose messages are hashed by a warp each (MsgGroup), the long
// ones apart: up to a warp a scheduler.  1024 verified messages of 2000 B take
// 1.068 ms that way, 1.056 in threads and two-warp blocks.
inline bool group_messages(uint64_t count) { return count <= 4ull * device_sms(); }

// finish key generation: sk.ROOT = pk.ROOT = top root, pk.PUB_SEED = sk.PUB_SEED
template <int n>
__global__ void k_keygen_finish(KeygenArgs A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.count) return;
    uint8_t *sk = A.sk + (uint64_t)i * 4 * n;
    uint8_t *pk = A.pk + (uint64_t)i * 2 * n;
    for (int j = 0; j < n; j++) {
        const uint8_t r = A.roots[(uint64_t)i * n + j];
        sk[3 * n + j] = r;
        pk[n + j] = r;
        pk[j] = sk[2 * n + j];
    }
}

template <class HF>
struct Family {
    static constexpr int W = HF::W, N = 4 * W;
    using TL = TlLanes<HF>;
    // Dynamic shared memory that k_leaf_chains asks for, to leave room on each
    // SM for the FORS trees beside it: with as many chain blocks as fit, robust
    // FORS at n = 32 (PRF and six-unit H) and the chains (three blocks of code)
    // took their SMs in turn.  With three chain blocks an SM, 1024 signatures
    // of 256f take 57.3 ms, 61.2 without, 100 of 256s 54.5 and 57.4; asking for
    // 56 or 44 KB gave 57.9 and 59.8 for the first.  128f-robust and
    // 192f-simple gained 1 % or less from a cap, 128f-simple nothing.
    static constexpr size_t kChainSmem = !HF::kShake && HF::kRobust && N == 32 ? 74u * 1024u : 0;

    static cudaError_t configure() {
        cudaError_t e;
        const int big = 200 * 1024;
        if ((e = cudaFuncSetAttribute(k_leaf_chains<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_leaves<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_leaf_tlen<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_fors_sign<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_trees<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_verify_ht<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if ((e = cudaFuncSetAttribute(k_verify_root<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if constexpr (kPersistVerify)
            if ((e = cudaFuncSetAttribute(k_verify_hyper<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big)))
                return e;
        if constexpr (HF::kShake)
            if ((e = cudaFuncSetAttribute(k_verify_item<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big)))
                return e;
        if ((e = cudaFuncSetAttribute(k_vsort_layer<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        if constexpr (!HF::kShake) {
            const void *blocks[] = {(const void *)k_verify_block<HF, 2>, (const void *)k_verify_block<HF, 4>,
                                    (const void *)k_verify_block<HF, 8>};
            for (const void *f : blocks)
                if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
            const void *layer[] = {(const void *)k_vsort_layer_group<HF, kGroupLanes>,
                                   (const void *)k_vsort_layer_group<HF, 4>};
            for (const void *f : layer)
                if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        }
        if ((e = cudaFuncSetAttribute(k_fors_pk<HF>, cudaFuncAttributeMaxDynamicSharedMemorySize, big))) return e;
        // Load every other kernel of the family now: with lazy module loading
        // a kernel's first launch loads it, and in a server that first launch
        // is a request's (one took ~50 ms of host time and held back every
        // queued request of its class).
        cudaFuncAttributes fa;
        const void *rest[] = {(const void *)k_sign_msg<HF>, (const void *)k_leaf_tstream<HF>,
                              (const void *)k_trees_lane<HF>, (const void *)k_fors_top<HF>, (const void *)k_share<HF>, (const void *)k_share_leaves<HF>,
                              (const void *)k_verify_msg<HF>, (const void *)k_verify_fors<HF>,
                              (const void *)k_verify_chains<HF>, (const void *)k_vsort_chains<HF>,
                              (const void *)k_vspec_cand<HF>,
                              (const void *)k_keygen_finish<N>};
        for (const void *f : rest)
            if ((e = cudaFuncGetAttributes(&fa, f))) return e;
        if constexpr (!HF::kShake) {
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_vspec_walk_group<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_key_mid<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_sign_msg_group<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_verify_msg_group<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_sign_msg_pair<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_verify_msg_pair<HF>))) return e;
        } else {
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_vsort_layer_warp<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_vspec_walk_warp<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_sign_msg_wide<HF>))) return e;
            if ((e = cudaFuncGetAttributes(&fa, (const void *)k_verify_msg_wide<HF>))) return e;
        }
        return cudaSuccess;
    }

    // SHA-256: the whole hypertree in one launch of blocks of I items
    // (spx_vblock.cuh).  More items a block fill its chain warps better but
    // leave its one T warp fewer lanes an item; few blocks an SM are bound by
    // a block's serial path, many by the SM.  Measured (ms, I = 2 / 4 / 8):
    // 128f, 301 items 0.92 / 0.85 / 1.08, 1024 items 1.39 / 1.23 / 1.11; 192f
    // 1.13 / 1.30 / 1.66, 2.27 / 1.96 / 1.76; 256f-robust 2.59 / 2.77 / 3.66,
    // 7.5 / 4.9 / 4.0.  (One block an item with its T lane behind the chains,
    // and warps that claim chains for up to 4 items, took 1.77 and 1.42 ms at
    // 301 items of 128f, 7.8 and 9.2 ms of 256f-robust.)
    static void verify_block(const SetParams &P, const VerifyArgs &A, cudaStream_t s) {
        if constexpr (!HF::kShake) {
            const uint64_t sms = (uint64_t)device_sms();
            if (A.count > 4 * sms) block_launch<8>(P, A, s);
            else if (N == 16 || A.count > 2 * sms) block_launch<4>(P, A, s);
            else block_launch<2>(P, A, s);
        }
    }
    template <int I>
    static void block_launch(const SetParams &P, const VerifyArgs &A, cudaStream_t s) {
        using VB = VerifyBlock<HF, I>;
        k_verify_block<HF, I><<<ceil_div(A.count, I), VB::kThreads, VB::words(P.hp) * 4, s>>>(P, A);
    }

    // SHAKE-256: the persistent verify kernel
    static constexpr bool kPersistVerify = HF::kShake;

    // one launch over the batch's whole hypertree: as many blocks as are
    // resident at once (or fewer for small batches); warps take items from
    // the counter as their slots free up
    static void verify_persistent(const SetParams &P, const VerifyArgs &A, const Tuning &tu, cudaStream_t s,
                                  PhaseTimer *pt) {
        if constexpr (kPersistVerify) {
            int wpb = tu.verify_block / 32;
            wpb = wpb < 1 ? 1 : (wpb > 4 ? 4 : wpb);
            const int sms = device_sms();
            int occ = 0;
            // Items per warp: one item's serial critical path (~d x 20
            // compressions) sets the time of a small batch, and a warp
            // holding several items runs their paths at a fraction of its
            // lanes each, so a batch first spreads to about 4 warps per SM
            // and only then packs up to verify_slots items per warp.
            const int gmax = tu.verify_slots < 1 ? 1 : (tu.verify_slots > 8 ? 8 : tu.verify_slots);
            int G = (int)ceil_div(A.count, 4ull * sms);
            G = G < 1 ? 1 : (G > gmax ? gmax : G);
            const size_t smem = (size_t)wpb * G * VerifyPolicy<HF>::slot_words(P.hp) * 4;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_verify_hyper<HF>, 32 * wpb, smem);
            if (occ < 1) occ = 1;
            const uint64_t want = ceil_div(A.count, (uint64_t)G * wpb);
            const uint64_t cap = (uint64_t)occ * (sms > 0 ? sms : 1);
            cudaMemsetAsync(A.ctr, 0, sizeof(uint32_t), s);
            const int claim_min = tu.verify_claim_min < 1 ? 1 : (tu.verify_claim_min > 32 ? 32 : tu.verify_claim_min);
            k_verify_hyper<HF><<<(unsigned)(want < cap ? want : cap), 32 * wpb, smem, s>>>(P, A, A.ctr, G, claim_min);
            CUSPX_MARK(pt, "k_verify_hyper", s);
        }
    }

    static void trees(const SetParams &P, const TreeArgs &T, const Tuning &tu, cudaStream_t s) {
        if (tu.tree_mode == 1 && P.hp <= 4) {
            const uint64_t threads = (uint64_t)T.count * T.nlayers;
            k_trees_lane<HF><<<ceil_div(threads, 128), 128, 0, s>>>(P, T);
            return;
        }
        const uint64_t per_warp = 2ull * (1u << P.hp) * W * 4;
        int wpb = (int)(48 * 1024 / per_warp);
        if (wpb > tu.tree_warps) wpb = tu.tree_warps;
        if (wpb < 1) wpb = 1;
        const uint64_t warps = (uint64_t)T.count * T.nlayers;
        k_trees<HF><<<ceil_div(warps, wpb), 32 * wpb, per_warp * wpb, s>>>(P, T);
    }

    // XMSS leaves.  With chain-end scratch: a thread per chain, then T_len, in
    // chunks of as many trees as the scratch holds.  Small sign batches
    // (`latency`) take several lanes a leaf for T_len up to two warps a
    // scheduler (128f, one signature 18 us, a thread a leaf 23 us; 37
    // signatures 35 / 23 us), larger ones the streaming kernel, whose threads
    // repeat nothing; robust SHA-256, whose lanes share out the mask blocks
    // too, takes them in every small batch (256f-robust, 37: 0.36 / 0.94 ms).
    // Without scratch (ends_trees 0): a thread per leaf (k_leaves).
    static void leaves(const SetParams &P, LeafArgs L, const Tuning &tu, cudaStream_t s, PhaseTimer *pt,
                       uint32_t ends_trees, bool latency) {
        const uint64_t trees = (uint64_t)L.count * L.nlayers;
        if (ends_trees == 0) {
            const int b = tu.leaf_block;
            k_leaves<HF><<<ceil_div(trees << P.hp, b), b, (size_t)b * HF::kSmemWords * 4, s>>>(P, L);
            CUSPX_MARK(pt, "k_leaves", s);
            return;
        }
        constexpr int LEN = 2 * N + 3;
        if (HF::kShake || !HF::kRobust) latency = latency && (trees << P.hp) * TL::kLanes <= 256ull * device_sms();
        L.interleaved = !latency;
        for (uint64_t t = 0; t < trees; t += ends_trees) {
            L.tree0 = (uint32_t)t;
            L.trees = (uint32_t)(trees - t < ends_trees ? trees - t : ends_trees);
            const uint64_t nl = (uint64_t)L.trees << P.hp;
            const uint32_t blocks = ceil_div(nl * LEN, 128);
            // from a few rounds of capped blocks on; one signature of 256f, 142
            // blocks, takes 0.41 ms capped and 0.35 not, and key generation has
            // no FORS trees to make room for
            const bool cap = L.work && blocks >= 16u * (uint32_t)device_sms();
            k_leaf_chains<HF><<<blocks, 128, cap ? kChainSmem : 0, s>>>(P, L);
            CUSPX_MARK(pt, "k_leaf_chains", s);
            if (latency) {
                k_leaf_tlen<HF><<<ceil_div(nl, TL::kPerBlock), TL::kThreads, TL::smem(), s>>>(P, L);
                CUSPX_MARK(pt, "k_leaf_tlen", s);
            } else {
                k_leaf_tstream<HF><<<ceil_div(nl, 128), 128, 0, s>>>(P, L);
                CUSPX_MARK(pt, "k_leaf_tstream", s);
            }
        }
    }

    // log2 of the lanes per FORS tree: tu.fors_lanes_log2, more where the trees
    // would leave SMs idle.  Within a warp, until the launch has 4 warps a
    // scheduler (beyond, the shuffle levels' idle lanes cost more than the
    // occupancy gives); with node scratch, tall trees over more lanes until it
    // has 16, several rounds of blocks, since a lane of a tall tree runs for
    // milliseconds and a part-empty last round is lost.
    static int fors_lanes(const SetParams &P, uint64_t trees, const Tuning &tu, uint64_t nodes) {
        const uint64_t sm = (uint64_t)device_sms();
        int g = tu.fors_lanes_log2 < P.a ? tu.fors_lanes_log2 : P.a;
        while (g < kForsWarpLanes && g < P.a && (trees << g) < sm * 512) g++;
        if (g == kForsWarpLanes)
            while (g < kForsMaxLanes && g < P.a && (trees << g) < sm * 2048 && (trees << (g + 1)) <= nodes) g++;
        return g;
    }

    static bool latency_mapping(uint32_t count, const Tuning &tu) {
        return count <= (uint32_t)tu.chain_mode_max && count <= kChainModeItems;
    }

    // First layer whose trees are looked for among the items (0: none).  A
    // layer of 8 trees per item still saves about 6% of its work if all items
    // have one key; the two memsets, k_share and k_share_leaves take 21 us at
    // 301 items and 25 to 50 from 1024 to 4096, so batches of the latency
    // mapping go without.
    static int share_layer(const SetParams &P, uint32_t count, const Tuning &tu, const ShareArgs &S) {
        if (!S.tab || count <= 64 || latency_mapping(count, tu)) return 0;
        return shared_layer0(P, count);
    }

    static void sign(const SetParams &P, SignArgs A, const Tuning &tu, cudaStream_t s, PhaseTimer *pt,
                     uint64_t long_msg, const StreamFork *fk) {
        if (A.count == 0) return;
        bool grouped = false;
        if constexpr (!HF::kShake) {
            grouped = group_messages(A.count);
            if (grouped) k_sign_msg_group<HF><<<A.count, 32, 0, s>>>(P, A, long_msg);
        }
        if (!grouped) k_sign_msg<HF><<<ceil_div(A.count, 128), 128, 0, s>>>(P, A, long_msg);
        CUSPX_MARK(pt, "k_sign_msg", s);
        if (long_msg) {   // messages of >= long_msg bytes: two warps per 32 (SHA-256), a warp each (SHAKE)
            if constexpr (!HF::kShake) {
                k_sign_msg_pair<HF><<<ceil_div(A.count, 32), 64, 0, s>>>(P, A, long_msg);
                CUSPX_MARK(pt, "k_sign_msg_pair", s);
            } else {
                k_sign_msg_wide<HF><<<ceil_div(A.count, 4), 128, 0, s>>>(P, A, long_msg);
                CUSPX_MARK(pt, "k_sign_msg_wide", s);
            }
        }
        // (k_leaves computes every item's trees)
        if (tu.chain_mode_max <= 0 && A.count <= kChainModeItems) A.ends_trees = 0;
        A.share.layer0 = A.ends_trees ? share_layer(P, A.count, tu, A.share) : 0;
        if (A.share.layer0) {
            const int tabs = P.d - A.share.layer0 + 1;
            A.share.mask = share_table(A.count) - 1;
            cudaMemsetAsync(A.share.cnt, 0, 16, s);
            cudaMemsetAsync(A.share.tab, 0, (size_t)tabs * (A.share.mask + 1) * 4, s);
            cudaMemsetAsync(A.share.recs, 0, ((size_t)(tabs - 1) * A.count << P.hp) * 4, s);
            k_share<HF><<<ceil_div((uint64_t)tabs * A.count, 128), 128, 0, s>>>(P, A);
            k_share_leaves<HF><<<ceil_div((uint64_t)(tabs - 1) * A.count, 128), 128, 0, s>>>(P, A);
            CUSPX_MARK(pt, "k_share", s);
        }
        const bool split = fk && !pt;
        cudaStream_t sf = split ? fk->side : s;
        if (split) {
            cudaEventRecord(fk->fork, s);
            cudaStreamWaitEvent(sf, fk->fork, 0);
        }
        {
            const int b = tu.fors_block;
            const uint64_t trees = (uint64_t)A.count * P.k;
            const int g = fors_lanes(P, trees, tu, A.fors_nodes ? A.fors_lanes : 0);
            k_fors_sign<HF><<<ceil_div(trees << g, b), b, (size_t)b * (P.a - g + 1) * W * 4, sf>>>(P, A, g);
            CUSPX_MARK(pt, "k_fors_sign", s);
            if (g > kForsWarpLanes) {
                const unsigned tb = g > 8 ? 256u : 1u << (g - 1);
                k_fors_top<HF><<<(unsigned)trees, tb, (size_t)W * 4 << g, sf>>>(P, A, g);
                CUSPX_MARK(pt, "k_fors_top", s);
            }
            k_fors_pk<HF><<<ceil_div(A.count, TL::kPerBlock), TL::kThreads, TL::smem(), sf>>>(P, A);
            CUSPX_MARK(pt, "k_fors_pk", s);
        }
        if (split) cudaEventRecord(fk->join, sf);
        {
            LeafArgs L{A.count, 0, P.d, A.sk, A.work, A.leaves, A.chains, A.ends, 0, 0, false, A.share, nullptr};
            leaves(P, L, tu, s, pt, A.ends_trees, latency_mapping(A.count, tu));
        }
        {
            TreeArgs T{A.count, 0, P.d, A.sk, A.work, A.leaves, A.roots, A.sig, A.share, nullptr};
            trees(P, T, tu, s);
            CUSPX_MARK(pt, "k_trees", s);
        }
        if (split) cudaStreamWaitEvent(s, fk->join, 0);
        k_sign_finish<HF><<<A.count, 128, 0, s>>>(P, A);
        CUSPX_MARK(pt, "k_sign_finish", s);
    }

    static constexpr uint32_t kLayerSmem = 200u * 1024u;   // the shared-memory limit configure() sets

    // SHA-256: batches of up to kGroupItems items run the layer kernel with
    // kGroupLanes lanes an item (spx_vgroup.cuh), one item group: the lanes
    // shorten the serial path (128f, 301 items: 0.92 ms a batch, against 1.33
    // with a thread an item), but all repeat its rounds, which costs a third
    // more issue slots, so larger batches take a thread an item and hide its
    // latency behind other item groups' chains (128f, lanes / thread: 2048
    // items 1.48 / 1.59 ms, 4096 2.45 / 2.22 ms; 192f 2.25 / 2.40, 3.65 / 3.29;
    // robust, whose H masks the lanes share out: 4096 items of 192f 6.6 / 8.0
    // ms, of 256s 5.0 / 5.2 ms, 8192 of 256s 10.4 / 9.7 ms).  32, 4 or 2 lanes
    // are slower than 8 from 301 to 2048 items but for 2 at 2048 (1.40 ms).
    // SHAKE-256: a warp an item, with the masks of robust sets squeezed by
    // threads of the chain launch (256f, warp / thread an item: 301 items 2.30
    // / 3.47 ms, 2048 5.76 / 6.00, 4096 9.9 / 9.1; 256f-robust 3.44 / 6.27,
    // 2048 items 9.8 / 12.0, 8192 34.9 / 34.9); one item group up to 4 items
    // an SM (128s-robust, 1024 items: 1.76 ms in one, 2.06 in four).
    static constexpr int kGroupLanes = 8;
    static constexpr uint32_t kGroupItems = HF::kShake ? (HF::kRobust ? 8192 : 2048) : (HF::kRobust ? 4096 : 2048);

    // SHA-256 batches of several item groups with lanes in the layer kernel as
    // well: it then ends before the other groups' chains do, and still leaves
    // them more of the SMs than 8 lanes would.  Returns the lanes an item (0:
    // none of these batches) and how many groups at most.  Simple f sets, 4
    // lanes: 128f 2048 items 1.384 ms (one group of 8 lanes 1.461), 4096 2.161
    // (a thread an item 2.20), 8192 3.586 / 3.649, but 12000 4.97 / 4.85; 192f
    // 3000 items 2.76 / 3.03, 5000 3.86 / 3.89, 6500 4.52 / 4.71, 8192 5.44 / 5.53
    // (8193, a thread an item: 5.54); 256f 3000 2.95 / 3.22, but 4096 3.77 / 3.68; the
    // s sets, whose layers are few, lose (128s, 4096: 0.90 / 0.86).  Robust
    // sets, whose H masks the lanes share out, in two groups, 8 lanes at n = 32
    // (256f 3000 items 6.69 / 7.22, 8192 16.6 / 17.9; 256s 3000 3.51 / 3.89,
    // but 2048 2.76 / 2.62) and 4 at n < 32 (192f 6000 items 8.80 / 10.3, 12000
    // 17.1 / 18.8; 128f 8192 7.30 / 7.73, but 4096 4.39 / 4.11; 192s 4200 2.56
    // / 3.30).  Their gain shrinks with the batch but had not ended at the largest
    // measured (192f, 65536 items: 93.8 / 96.6 ms; 256f 49152: 101.0 / 102.8; 128s
    // 65536: 19.3 / 20.1), so they have no upper end.
    static int side_lanes(const SetParams &P, uint32_t count, int &groups) {
        if (HF::kShake) return 0;
        if (!HF::kRobust) {
            if (P.d <= 8 || count < 1500 || count > (N < 32 ? 8192u : 3072u)) return 0;
            if (groups > 4) groups = 4;   // 128f, 4096 items: 2.14 ms, 2.17 in 6 and 2.21 in 8
            return 4;
        }
        if (N == 32 ? count < 3000 : count <= 4096) return 0;
        groups = 2;
        return N == 32 ? 8 : 4;
    }

    // verify_mode 3: per group of items, T_k then per layer the sorted
    // chains and the layer roots (spx_vsort.cuh).  Groups run on their own
    // streams; a group's chain kernel of layer L starts after the previous
    // group's, so the groups keep an offset and one group's serial layer
    // kernel overlaps the next group's chains.  With per-kernel timing on
    // every group runs on s.
    static void verify_sorted(const SetParams &P, const VerifyArgs &A, const Tuning &tu, cudaStream_t s,
                              PhaseTimer *pt, const VerifyLists &V, const VerifyFork *vf) {
        constexpr int LEN = 2 * N + 3;
        const int gmax = pt || !vf ? 1 : vf->sides + 1;
        int G = tu.verify_groups < 1 ? 1 : tu.verify_groups;
        if (G > gmax) G = gmax;
        int most = G;
        const int side = G > 1 ? side_lanes(P, A.count, most) : 0;
        if (G > most) G = most;
        const bool grouped = side > 0 || (A.count <= kGroupItems && (!HF::kShake || !HF::kRobust || V.masks));
        if (!side && grouped && (!HF::kShake || A.count <= 4u * (uint32_t)device_sms())) G = 1;
        if ((uint32_t)G > A.count) G = (int)A.count;
        const uint32_t per = (A.count + G - 1) / G;
        G = (int)((A.count + per - 1) / per);
        // thread per item in the layer kernel, whose slots must fit the
        // 200 KiB of shared memory configured for it (32 threads fit for
        // every set: SHAKE-256f-robust needs 176 KiB)
        int b = tu.verify_block;
        while (b > 32 && VsortSmem<HF>::bytes(P, (uint32_t)b) > kLayerSmem) b /= 2;
        auto layer = [&](int L, uint32_t first, uint32_t n, int g, cudaStream_t st) {
            if constexpr (HF::kShake) {
                if (grouped) {
                    k_vsort_layer_warp<HF><<<ceil_div(n, 4), 128, 0, st>>>(P, A, V, L, first, n, g);
                    return;
                }
            }
            if constexpr (!HF::kShake) {
                if (side == 4) {
                    constexpr int kItems = 16;
                    k_vsort_layer_group<HF, 4>
                        <<<ceil_div(n, kItems), 64, kItems * ShaGroup<HF>::kStride * 4, st>>>(P, A, V, L, first, n, g);
                    return;
                }
                if (grouped) {
                    constexpr int kItems = 64 / kGroupLanes;
                    k_vsort_layer_group<HF, kGroupLanes>
                        <<<ceil_div(n, kItems), 64, kItems * ShaGroup<HF>::kStride * 4, st>>>(P, A, V, L, first, n, g);
                    return;
                }
            }
            k_vsort_layer<HF><<<ceil_div(n, b), b, VsortSmem<HF>::bytes(P, (uint32_t)b), st>>>(P, A, V, L, first, n, g);
        };
        cudaMemsetAsync(V.cnt, 0, (size_t)G * P.d * 16 * sizeof(uint32_t), s);
        cudaStream_t gs[VerifyFork::kMaxGroups];
        gs[0] = s;
        if (G > 1) cudaEventRecord(vf->fork, s);
        for (int g = 1; g < G; g++) {
            gs[g] = vf->side[g - 1];
            cudaStreamWaitEvent(gs[g], vf->fork, 0);
        }
        auto first = [&](int g) { return (uint32_t)g * per; };
        auto items = [&](int g) { return g + 1 < G ? per : A.count - (uint32_t)g * per; };
        for (int g = 0; g < G; g++) {
            k_verify_fors<HF><<<ceil_div((uint64_t)items(g) * P.k, 128), 128, 0, gs[g]>>>(P, A, first(g), items(g));
            CUSPX_MARK(pt, "k_verify_fors", s);
            layer(-1, first(g), items(g), g, gs[g]);
            CUSPX_MARK(pt, "k_vsort_layer", s);
        }
        for (int L = 0; L < P.d; L++) {
            for (int g = 0; g < G; g++) {
                if (g > 0) cudaStreamWaitEvent(gs[g], vf->chain[g - 1], 0);
                const uint32_t mb = grouped && HF::kShake && HF::kRobust ? ceil_div(2ull * items(g), 128) : 0;
                k_vsort_chains<HF><<<mb + ceil_div((uint64_t)items(g) * LEN, 128), 128, 0, gs[g]>>>(
                    P, A, V, L, first(g), g, items(g), mb);
                CUSPX_MARK(pt, "k_vsort_chains", s);
                if (g + 1 < G) cudaEventRecord(vf->chain[g], gs[g]);
                layer(L, first(g), items(g), g, gs[g]);
                CUSPX_MARK(pt, "k_vsort_layer", s);
            }
        }
        for (int g = 1; g < G; g++) {
            cudaEventRecord(vf->join[g - 1], gs[g]);
            cudaStreamWaitEvent(s, vf->join[g - 1], 0);
        }
    }

    static void verify(const SetParams &P, const VerifyArgs &A, const Tuning &tu, cudaStream_t s, PhaseTimer *pt,
                       uint64_t long_msg, const VerifyLists *vl, const VerifyFork *vf) {
        if (A.count == 0) return;
        bool grouped = false;
        if constexpr (!HF::kShake) {
            grouped = group_messages(A.count);
            if (grouped) k_verify_msg_group<HF><<<A.count, 32, 0, s>>>(P, A, long_msg);
        }
        if (!grouped) k_verify_msg<HF><<<ceil_div(A.count, 128), 128, 0, s>>>(P, A, long_msg);
        CUSPX_MARK(pt, "k_verify_msg", s);
        if (long_msg) {
            if constexpr (!HF::kShake) {
                k_verify_msg_pair<HF><<<ceil_div(A.count, 32), 64, 0, s>>>(P, A, long_msg);
                CUSPX_MARK(pt, "k_verify_msg_pair", s);
            } else {
                k_verify_msg_wide<HF><<<ceil_div(A.count, 4), 128, 0, s>>>(P, A, long_msg);
                CUSPX_MARK(pt, "k_verify_msg_wide", s);
            }
        }
        const bool spec = tu.verify_mode != 3 && tu.verify_spec_max > 0 && A.count <= (uint32_t)tu.verify_spec_max &&
                          vl && vl->cand && A.count <= vl->cand_items &&
                          P.len1 == 2 * N && P.len2 == 3;
        const bool by_size = tu.verify_sorted_min > 0 && A.count >= (uint32_t)tu.verify_sorted_min;
        const bool direct = vl && vl->direct;   // each launch is a host launch (serving)
        const bool item = A.count <= (uint32_t)(tu.verify_item_max > 0 ? tu.verify_item_max : 0) ||
                          (HF::kShake && direct && A.count <= 128);
        // launches of their own for the layers pay above 4 items an SM for
        // SHA-256 (128f, 700 items: 0.97 ms, fused 1.09) and at every size for
        // SHAKE-256 (256f, 64 items: 2.29 ms, one item per block 2.85; 301
        // items 2.30, persistent 3.11), unless sorted_min is 0
        const bool layers = tu.verify_sorted_min > 0 && tu.verify_mode >= 2 && !direct && !spec &&
                            (HF::kShake || A.count > 4u * (uint32_t)device_sms());
        const bool sorted = (tu.verify_mode == 3 || by_size || layers) && vl && vl->tasks &&
                            vl->stride >= (uint64_t)A.count * (2 * N + 3) && A.count < (1u << 25) &&
                            VsortSmem<HF>::bytes(P, 32) <= kLayerSmem && P.len1 == 2 * N && P.len2 == 3 && !item;
        if (sorted) {   // FORS per item group, beside the other groups' layers
            verify_sorted(P, A, tu, s, pt, *vl, vf);
            return;
        }
        if (spec) {
            // tiny batches: every chain run from every start step, then the
            // serial walk over T_len and the auth paths alone (spx_vsort.cuh)
            // (the chain runs beside the FORS roots, on a side stream)
            constexpr int LEN = 2 * N + 3;
            const bool side = !pt && vf && vf->sides > 0;
            cudaStream_t cs = side ? vf->side[0] : s;
            if (side) {
                cudaEventRecord(vf->fork, s);
                cudaStreamWaitEvent(cs, vf->fork, 0);
            }
            const uint64_t mask_tasks = HF::kShake && HF::kRobust ? 2ull * A.count * P.d : 0;
            k_vspec_cand<HF><<<ceil_div(16ull * A.count * P.d * LEN + mask_tasks, 128), 128, 0, cs>>>(
                P, A, vl->cand, vl->cand_masks);
            CUSPX_MARK(pt, "k_vspec_cand", s);
            k_verify_fors<HF><<<ceil_div((uint64_t)A.count * P.k, 128), 128, 0, s>>>(P, A, 0, A.count);
            CUSPX_MARK(pt, "k_verify_fors", s);
            if (side) {
                cudaEventRecord(vf->join[0], cs);
                cudaStreamWaitEvent(s, vf->join[0], 0);
            }
            if constexpr (!HF::kShake)
                k_vspec_walk_group<HF><<<A.count, 32, ShaGroup<HF>::kWords * 4, s>>>(P, A, vl->cand);
            else
                k_vspec_walk_warp<HF><<<A.count, 32, 0, s>>>(P, A, vl->cand, vl->cand_masks);
            CUSPX_MARK(pt, "k_vspec_walk", s);
            return;
        }
        k_verify_fors<HF><<<ceil_div((uint64_t)A.count * P.k, 128), 128, 0, s>>>(P, A, 0, A.count);
        CUSPX_MARK(pt, "k_verify_fors", s);
        if constexpr (!HF::kShake) {
            if ((item || (tu.verify_mode >= 2 && A.ctr)) && P.hp <= 9) {
                verify_block(P, A, s);
                CUSPX_MARK(pt, "k_verify_block", s);
                return;
            }
        } else if (item && P.hp <= 9) {
            // small batches: one item per block (its serial path sets the time)
            constexpr int LEN = 2 * N + 3, CW = (LEN + 31) / 32;
            // one slot and the prefetched auth path of the next layer
            const size_t smem = ((size_t)VerifyPolicy<HF>::slot_words(P.hp) + (size_t)P.hp * W) * 4;
            k_verify_item<HF><<<A.count, 32 * (CW + 1), smem, s>>>(P, A);
            CUSPX_MARK(pt, "k_verify_item", s);
            return;
        } else if (tu.verify_mode >= 2 && A.ctr && P.hp <= 9) {
            verify_persistent(P, A, tu, s, pt);
            return;
        }
        const int b = tu.verify_block;
        if (tu.verify_mode == 1) {
            k_verify_ht<HF><<<ceil_div(A.count, b), b, (size_t)b * HF::kSmemWords * 4, s>>>(P, A);
            CUSPX_MARK(pt, "k_verify_ht", s);
            return;
        }
        constexpr int LEN = 2 * N + 3;
        const int pw = tu.chains_per_warp;
        const uint64_t warps = ((uint64_t)A.count * LEN + pw - 1) / pw;
        for (int L = -1; L < P.d; L++) {
            if (L >= 0) {
                k_verify_chains<HF><<<ceil_div(warps, 4), 128, 0, s>>>(P, A, L, pw);
                CUSPX_MARK(pt, "k_verify_chains", s);
            }
            k_verify_root<HF><<<ceil_div(A.count, b), b, (size_t)b * HF::kSmemWords * 4, s>>>(P, A, L);
            CUSPX_MARK(pt, "k_verify_root", s);
        }
    }

    static void keygen(const SetParams &P, const KeygenArgs &K, const Tuning &tu, cudaStream_t s, PhaseTimer *pt) {
        if (K.count == 0) return;
        KeyRef kr{K.sk, nullptr, (uint32_t)(4 * N)};
        if constexpr (!HF::kShake) {
            k_key_mid<HF><<<ceil_div(K.count, 128), 128, 0, s>>>(kr, K.count, K.mids);
            CUSPX_MARK(pt, "k_key_mid", s);
        }
        LeafArgs L{K.count, P.d - 1, 1, kr, nullptr, K.leaves, nullptr, K.ends, 0, 0, false, {}, K.mids};
        leaves(P, L, tu, s, pt, tu.chain_mode_max > 0 ? K.ends_trees : 0, false);
        TreeArgs T{K.count, P.d - 1, 1, kr, nullptr, K.leaves, K.roots, nullptr, {}, K.mids};
        trees(P, T, tu, s);
        CUSPX_MARK(pt, "k_trees", s);
        k_keygen_finish<N><<<ceil_div(K.count, 128), 128, 0, s>>>(K);
        CUSPX_MARK(pt, "k_keygen_finish", s);
    }

    static FamilyOps ops() {
        FamilyOps o;
        o.configure = &configure;
        o.sign = &sign;
        o.verify = &verify;
        o.keygen = &keygen;
        o.smem_words = HF::kSmemWords;
        return o;
    }
};

}  // namespace cuspx
