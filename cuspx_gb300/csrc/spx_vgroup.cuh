// spx_vgroup.cuh -- verify: T_l and auth paths by a group of lanes per item.
//
// SHA-256.  What is serial in a verify layer is T_len over the len chain ends (10
// compressions at n = 16, 35 at n = 32) and the auth path.  A compression's
// chaining goes through its rounds alone: the message schedules of all of
// T_len's blocks are independent.  Here the G lanes of an item compute them
// side by side (lane g those of blocks g, g + G, ...) into shared memory,
// W_t + K_t, and then all run the rounds, the same ones in every lane, from
// broadcast reads.  A warp alone on its SM takes 31 cycles a round that way,
// against ~46 with the schedule in between, and beside other warps the serial
// path issues 15 instead of 24 instructions a round.  Robust sets' bitmasks
// of the auth path (and of T_k) depend on addresses alone and are computed by
// the lanes side by side too.
#pragma once
#include "spx_kernels.cuh"

namespace cuspx {

template <class HF>
struct ShaGroup {
    static constexpr int W = HF::W, N = 4 * W, LEN = 2 * N + 3, LEN1 = 2 * N;
    static constexpr int blocks(int m) { return (22 + m * N + 9 + 63) / 64; }
    static constexpr int NB = blocks(LEN);        // no set's T_k is longer
    static constexpr int NBP = NB | 1;            // row of kw: an odd stride spreads the lanes' stores over the banks
    static constexpr int kMaskH = HF::kRobust ? (2 * W + 7) / 8 : 0;   // mask blocks of an H
    static constexpr int kMaxHp = 9;              // tallest subtree of any set
    // an item's shared words: kw[t * NBP + block], the H masks, the layer's message
    static constexpr int S_HM = 64 * NBP, S_ROOT = S_HM + kMaxHp * kMaskH * 8, kWords = S_ROOT + 8;
    // a stride of 4 mod 32 keeps the groups of a warp in different banks
    static constexpr int kStride = kWords + (36 - kWords % 32) % 32;

    // s <- compress(s, w) with each round's h + K + W made a round early and
    // the schedule a round ahead of its use: for a warp alone on its SM (the
    // walk of one 128f item 0.445 -> 0.432 ms against sha256_compress)
    SPX_DEV static void compress_ahead(uint32_t s[8], uint32_t w[16]) {
        uint32_t a = s[0], b = s[1], c = s[2], d = s[3], e = s[4], f = s[5], g = s[6], h = s[7];
        uint32_t hk = h + (w[0] + sha256_k(0));
#pragma unroll
        for (int i = 0; i < 64; i++) {
            const int t = i + 1;
            if (t >= 16 && t < 64)
                w[t & 15] = add_fma(w[t & 15], sha_sigma0(w[(t - 15) & 15]) + w[(t - 7) & 15] +
                                                   sha_sigma1(w[(t - 2) & 15]));
            const uint32_t nx = t < 64 ? g + (w[t & 15] + sha256_k(t & 63)) : 0u;
            const uint32_t S1 = sha_Sigma1(e), ch = (e & f) ^ (~e & g);
            const uint32_t S0 = sha_Sigma0(a), mj = (a & b) | (c & (a | b));
            const uint32_t t1 = hk + S1 + ch;
            hk = nx;
            h = g;
            g = f;
            f = e;
            e = add_fma(d, t1);
            d = c;
            c = b;
            b = a;
            a = t1 + (S0 + mj);
        }
        s[0] += a; s[1] += b; s[2] += c; s[3] += d; s[4] += e; s[5] += f; s[6] += g; s[7] += h;
    }

    // T_l of m values under ADRS pa into out, in every lane of the group; g
    // the lane's number in it.  ld(q): bytes 8q .. 8q + 7 of the values (memory
    // order), already xored with a robust set's mask unless `mask`.  Every lane
    // of the warp calls this, with the same m.
    template <int G, class LD>
    SPX_DEV static void tl(uint32_t out[W], uint32_t *S, uint32_t g, const KeyRegs<N> &key, const Adrs &pa, int m,
                           bool mask, LD ld) {
        const int nb = blocks(m), Q = m * N / 8;
        for (int j = (int)g; j < nb; j += G) {
            uint32_t v[18], w[16];   // v[i]: value word 16j - 6 + i (see Sha2::t_values)
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const int q = 8 * j - 3 + i;
                uint2 x = make_uint2(0u, 0u);
                if (q >= 0 && q < Q) x = ld((uint32_t)q);
                v[2 * i] = bswap32(x.x);
                v[2 * i + 1] = bswap32(x.y);
            }
            if (HF::kRobust && mask) {
#pragma unroll 1
                for (int b = 0; b < 3; b++) {   // mask blocks 2j - 1, 2j, 2j + 1
                    uint32_t x[8];
                    if (2 * j - 1 + b >= 0) HF::mask_block(x, key.pub, pa, (uint32_t)(2 * j - 1 + b));
#pragma unroll
                    for (int i = 0; i < 18; i++) {
                        const int p = 16 * j - 6 + i;
                        if (p >= 0 && p < m * W && (i + 2) / 8 == b) v[i] ^= x[(i + 2) % 8];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = __funnelshift_l(v[i + 1], v[i], 16);
            if (j == 0) {
#pragma unroll
                for (int i = 0; i < 5; i++) w[i] = pa.w[i];
                w[5] |= pa.w[5] & 0xffff0000u;
            }
            const int pad = 5 + m * W - 16 * j;   // stream word that holds the padding byte
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i == pad) w[i] |= 0x8000u;
            if (j == nb - 1) w[15] = (uint32_t)(64 + 22 + m * N) * 8u;
            sha256_schedule_kw<NBP>(S + j, w);
        }
        __syncwarp();
        uint32_t st[8];
#pragma unroll
        for (int i = 0; i < 8; i++) st[i] = key.mid[i];
#pragma unroll 1
        for (int j = 0; j < nb; j++) {
            if constexpr (HF::kRobust) sha256_compress_kw16<NBP>(st, S + j);   // beside mask blocks
            else sha256_compress_kw<NBP>(st, S + j);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = st[i];
    }

    // robust sets: the H masks of the layer's auth path into the item's
    // shared words, before climb; every lane of the warp calls this
    template <int G>
    SPX_DEV static void h_masks(uint32_t *S, uint32_t g, const KeyRegs<N> &key, int hp, Adrs ad, uint32_t idx) {
        if constexpr (HF::kRobust) {
            for (int t = (int)g; t < hp * kMaskH; t += G) {
                const int h = t / kMaskH;
                adrs_height(ad, h + 1);
                adrs_index(ad, idx >> (h + 1));
                uint32_t x[8];
                HF::mask_block(x, key.pub, ad, (uint32_t)(t % kMaskH));
#pragma unroll
                for (int i = 0; i < 8; i++) S[S_HM + t * 8 + i] = x[i];
            }
            __syncwarp();
        }
    }

    // root <- compute_root (utils.cu:94-135) of leaf `root` over the auth path
    // at auth; ad: the layer's HASHTREE address
    SPX_DEV static void climb(uint32_t root[W], const uint32_t *S, const KeyRegs<N> &key, int hp, Adrs ad, uint32_t idx,
                              const uint8_t *auth) {
        uint32_t nx[W];
        HF::load(nx, auth);
#pragma unroll 1
        for (int h = 0; h < hp; h++) {
            uint32_t in[2 * W], st[8];
            const bool right = (idx >> h) & 1u;
#pragma unroll
            for (int i = 0; i < W; i++) {
                in[i] = right ? nx[i] : root[i];
                in[W + i] = right ? root[i] : nx[i];
            }
            if (h + 1 < hp) HF::load(nx, auth + (uint64_t)(h + 1) * N);
            if constexpr (HF::kRobust) {
#pragma unroll
                for (int i = 0; i < 2 * W; i++) in[i] ^= S[S_HM + (h * kMaskH + i / 8) * 8 + i % 8];
            }
            adrs_height(ad, h + 1);
            adrs_index(ad, idx >> (h + 1));
#pragma unroll
            for (int i = 0; i < 8; i++) st[i] = key.mid[i];
#pragma unroll 1
            for (int b = 0; b < HF::template kBlocks<2 * W>; b++) {
                uint32_t w[16];
                HF::template core_block<2 * W>(w, ad, in, b);
                compress_ahead(st, w);
            }
#pragma unroll
            for (int i = 0; i < W; i++) root[i] = st[i];
        }
    }

    // checksum digits of a WOTS+ message (chain_lengths, wots.cu:84-166), 4 bits each
    SPX_DEV static uint32_t checksum(const uint32_t msg[W]) {
        uint32_t sum = 0;
#pragma unroll
        for (int i = 0; i < W; i++)
            sum += __dp4a((msg[i] & 0x0f0f0f0fu) + (msg[i] >> 4 & 0x0f0f0f0fu), 0x01010101u, 0u);
        return (15u * LEN1 - sum) << 4;
    }
    // digit c of the message whose words are in S[S_ROOT ..]
    SPX_DEV static uint32_t digit(const uint32_t *S, uint32_t csum, uint32_t c) {
        if (c < (uint32_t)LEN1) return S[S_ROOT + (c >> 3)] >> (28 - 4 * (c & 7)) & 15u;
        return csum >> (12 - 4 * (c - LEN1)) & 15u;
    }

    // The root of layer L of an item (L = -1: its FORS key), in every lane of
    // its group; auth: the layer's auth path.  Every lane of the warp calls this.
    template <int G, class LD>
    SPX_DEV static void layer_root(uint32_t root[W], const SetParams &P, uint32_t *S, uint32_t g, const KeyRegs<N> &key,
                                   uint64_t tree, uint32_t idx_leaf, const uint8_t *auth, int L, LD ld) {
        uint64_t tree_L = tree;
        uint32_t idx_L = idx_leaf;
        Adrs pa;
        adrs_zero(pa);
        if (L >= 0) {
            layer_index(P, tree, idx_leaf, L, tree_L, idx_L);
            adrs_layer(pa, L);
        }
        adrs_tree(pa, tree_L);
        adrs_keypair(pa, idx_L);
        adrs_type(pa, L < 0 ? ADDR_FORSPK : ADDR_WOTSPK);
        tl<G>(root, S, g, key, pa, L < 0 ? P.k : LEN, L < 0, ld);
        if (L < 0) return;
        Adrs ad;
        adrs_zero(ad);
        adrs_layer(ad, L);
        adrs_tree(ad, tree_L);
        adrs_type(ad, ADDR_HASHTREE);
        h_masks<G>(S, g, key, P.hp, ad, idx_L);
        climb(root, S, key, P.hp, ad, idx_L, auth);
    }
};

// ---------------------------------------------------------------------------
// SHA-256 message hashing, a warp per item, for small batches: the schedules
// of 32 blocks of a message are computed side by side, then every lane runs
// the rounds on them in turn.  What is a block by itself, the HMAC pads, MGF1's
// blocks and the key's midstate, goes through the same two pieces of code, a
// block a lane: with unrolled compressions of their own the kernel fetched
// enough code to be 2 us slower than threads at 33 B.  A warp alone is bound by
// the rounds' latency.  One message under 128f, against a thread (or from 1024
// B verified and 1536 B signed on, two warps): 33 B signed 92.9 -> 88.3 us, of
// 1024 B 144 -> 118, of 4000 B 226 -> 212; 1024 B verified 446 -> 434.
// ---------------------------------------------------------------------------
template <class HF>
struct MsgGroup {
    static constexpr int W = HF::W, N = 4 * W, NBP = 33;
    uint32_t kw[64 * NBP], pre[3 * W], dg[16];

    // with_prf: R <- PRF_msg (HMAC-SHA256(SK_PRF, optrand || m)).  Returns the
    // work record of H_msg = MGF1(SHA256(R || PK || m)) in every lane.  All
    // lanes of the warp call this with the same arguments.
    SPX_DEV SignWork run(const SetParams &P, uint32_t R[W], bool with_prf, const uint32_t skprf[W],
                         const uint32_t opt[W], const uint32_t pk[2 * W], const uint8_t *m, uint64_t mlen,
                         uint32_t lane) {
        uint32_t st[8], outer[8];
        sha256_iv(st);
        sha256_iv(outer);
        // 0 ipad and opad, 1 optrand || m, 2 inner digest, 3 R || PK || m, 4 MGF1 and PUB_SEED
#pragma unroll 1
        for (int ph = with_prf ? 0 : 3; ph < 5; ph++) {
            const bool own = !(ph & 1);   // a block a lane
            const uint32_t np = ph == 1 ? W : 3 * W;
            if (!own && lane == 0) {
#pragma unroll
                for (int i = 0; i < W; i++) {
                    pre[i] = ph == 1 ? opt[i] : R[i];
                    pre[W + i] = pk[i];
                    pre[2 * W + i] = pk[W + i];
                }
            }
            __syncwarp();
            const uint64_t bytes = 4 * np + mlen;
            const uint64_t bits = ((ph == 1 ? 64 : 0) + bytes) * 8;
            const uint64_t nb = own ? 1 : (bytes + 9 + 63) / 64;
            for (uint64_t b0 = 0; b0 < nb; b0 += 32) {
                uint32_t w[16];
                if (own) {
                    const uint32_t pad = lane == 0 ? 0x36363636u : 0x5c5c5c5cu;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const uint32_t kp = (i < W ? skprf[i < W ? i : 0] : 0u) ^ pad;
                        const uint32_t pb = i < W ? pk[i < W ? i : 0] : 0u;
                        w[i] = ph == 0 ? kp : (ph == 4 && lane == 31 ? pb : st[i]);
                    }
#pragma unroll
                    for (int i = 8; i < 16; i++) {
                        const uint32_t v2 = i == 8 ? 0x80000000u : (i == 15 ? (64 + 32) * 8 : 0u);
                        const uint32_t v4 = i == 8 ? lane : (i == 9 ? 0x80000000u : (i == 15 ? 36 * 8 : 0u));
                        w[i] = ph == 0 ? pad : (ph == 2 ? v2 : (lane == 31 ? 0u : v4));
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++) st[i] = outer[i];
                    if (ph != 2) sha256_iv(st);
                } else {
                    const uint64_t b = b0 + lane;
                    if (b < nb) {
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const uint64_t g = 16 * b + i;
                            w[i] = g < np ? pre[g] : HF::msg_word(m, mlen, g - np);
                        }
                        if (b == nb - 1) {
                            w[14] = (uint32_t)(bits >> 32);
                            w[15] = (uint32_t)bits;
                        }
                    }
                }
                if (own || b0 + lane < nb) sha256_schedule_kw<NBP>(kw + lane, w);
                __syncwarp();
                const uint32_t n = nb - b0 < 32 ? (uint32_t)(nb - b0) : 32u;
#pragma unroll 1
                for (uint32_t j = 0; j < n; j++) sha256_compress_kw<NBP>(st, kw + (own ? lane : j));
                __syncwarp();
            }
            if (ph == 0) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    outer[i] = __shfl_sync(0xffffffffu, st[i], 1);
                    st[i] = __shfl_sync(0xffffffffu, st[i], 0);
                }
            } else if (ph == 2) {
#pragma unroll
                for (int i = 0; i < W; i++) R[i] = st[i];
                sha256_iv(st);
            }
        }
        if (lane < 2) {
#pragma unroll
            for (int i = 0; i < 8; i++) dg[8 * lane + i] = bswap32(st[i]);
        }
        __syncwarp();
        SignWork wk = work_indices(P, reinterpret_cast<const uint8_t *>(dg));
#pragma unroll
        for (int i = 0; i < 8; i++) wk.mid[i] = __shfl_sync(0xffffffffu, st[i], 31);
        return wk;
    }
};

template <class HF>
__global__ void __launch_bounds__(32) k_sign_msg_group(SetParams P, SignArgs A, uint64_t long_msg) {
    constexpr int W = HF::W, N = 4 * W;
    __shared__ MsgGroup<HF> S;
    const uint32_t i = blockIdx.x, lane = threadIdx.x;
    if (long_msg && A.msg.len[i] >= long_msg) return;   // k_sign_msg_pair hashes it
    const uint8_t *sk = A.sk.row(i);
    uint32_t skprf[W], opt[W], pk[2 * W], R[W];
    HF::load(skprf, sk + N);
    HF::load(pk, sk + 2 * N);
    HF::load(pk + W, sk + 3 * N);
#pragma unroll
    for (int j = 0; j < W; j++) opt[j] = 0xadadadadu;   // the reference's fixed optrand (sign.cu:1950-1954)
    if (A.optrand) HF::load(opt, A.optrand + (uint64_t)i * N);
    const SignWork wk = S.run(P, R, true, skprf, opt, pk, A.msg.base + A.msg.off[i], A.msg.len[i], lane);
    if (lane == 0) {
        HF::store(A.sig + (uint64_t)i * P.sig_bytes, R);
        A.work[i] = wk;
    }
}

template <class HF>
__global__ void __launch_bounds__(32) k_verify_msg_group(SetParams P, VerifyArgs A, uint64_t long_msg) {
    constexpr int W = HF::W, N = 4 * W;
    __shared__ MsgGroup<HF> S;
    const uint32_t i = blockIdx.x, lane = threadIdx.x;
    if (A.siglen && A.siglen[i] != (uint64_t)P.sig_bytes) {   // reject without hashing (sign.cu:3063-3065)
        if (lane == 0) {
            SignWork w = {};
            w.flags = 1;
            A.work[i] = w;
        }
        return;
    }
    if (long_msg && A.msg.len[i] >= long_msg) return;   // k_verify_msg_pair hashes it
    const uint8_t *pkb = A.pk.row(i);
    uint32_t R[W], pk[2 * W];
    HF::load(R, A.sig + (uint64_t)i * A.sig_stride);
    HF::load(pk, pkb);
    HF::load(pk + W, pkb + N);
    const SignWork wk = S.run(P, R, false, R, R, pk, A.msg.base + A.msg.off[i], A.msg.len[i], lane);
    if (lane == 0) A.work[i] = wk;
}

// ---------------------------------------------------------------------------
// SHAKE-256 T_l and auth paths by a warp per item: the sponge state spread
// over the warp (warp_keccak_f1600), lane j < 17 absorbing lane j of each
// block.  A permutation is 1,080 instructions of the warp instead of 4,300 of
// one thread: 3.0 us against 4.3 for a warp alone on its SM, and a quarter of
// the time beside chain warps that share its scheduler.  Robust sets' masks
// depend on addresses alone: threads of the chain kernels squeeze them
// (shake_mask_task) while the chains run.
// ---------------------------------------------------------------------------
template <class HF>
struct ShakeGroup {
    static constexpr int W = HF::W, N = 4 * W, NL = N / 8, LEN = 2 * N + 3, LEN1 = 2 * N, PL = NL + 4;
    // 64-bit words of a layer's masks of one item: T_len's, then 2n bytes per H
    static __host__ __device__ constexpr int mask_lanes(int hp) { return LEN * NL + hp * 2 * NL; }

    // lane p of PUB_SEED || ADRS (p < PL)
    SPX_DEV static uint64_t prefix(const uint8_t *pk, const Adrs &a, uint32_t p) {
        uint64_t al[4];
        adrs_lanes(a, al);
        uint64_t x = p < (uint32_t)NL ? reinterpret_cast<const uint64_t *>(pk)[p < (uint32_t)NL ? p : 0] : 0ull;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (p == (uint32_t)(NL + i)) x = al[i];
        return x;
    }

    // T_l of m values under ADRS pa: lane i < NL returns lane i of the result.
    // ld(q): lane q of the values, masked already unless `mask`.
    template <class LD>
    SPX_DEV static uint64_t tl(const KeccakLane &k, uint32_t lane, const uint8_t *pk, const Adrs &pa, int m, bool mask,
                               LD ld) {
        const int Q = m * NL, nb = (PL + Q) / 17 + 1;
        const uint64_t pre = lane < (uint32_t)PL ? prefix(pk, pa, lane) : 0ull;
        auto block = [&](int b) -> uint64_t {
            const int q = 17 * b + (int)lane - PL;
            if (lane >= 17) return 0ull;
            if (q < 0) return pre;
            uint64_t x = q < Q ? ld((uint32_t)q) : (q == Q ? 0x1Full : 0ull);
            if (b == nb - 1 && lane == 16) x ^= 0x8000000000000000ull;
            return x;
        };
        uint64_t a = 0, ms = 0, last = 0, nxt = block(0);
        if (HF::kRobust && mask) {   // SHAKE256(PUB_SEED || ADRS), squeezed a block ahead
            ms = pre ^ (lane == (uint32_t)PL ? 0x1Full : 0ull) ^ (lane == 16 ? 0x8000000000000000ull : 0ull);
        }
#pragma unroll 1
        for (int b = 0; b < nb; b++) {
            uint64_t cur = nxt;
            if (b + 1 < nb) nxt = block(b + 1);
            if (HF::kRobust && mask) {
                // block b's value lanes take mask lanes 17b - PL ..: the end of
                // mask block b - 1, then block b
                warp_keccak_f1600(ms, k, lane);
                const uint64_t hi = shfl64(last, (lane + 17 - PL) & 31), lo = shfl64(ms, (lane - PL) & 31);
                const int q = 17 * b + (int)lane - PL;
                if (lane < 17 && q >= 0 && q < Q) cur ^= lane < (uint32_t)PL ? hi : lo;
                last = ms;
            }
            a ^= cur;
            warp_keccak_f1600(a, k, lane);
        }
        return a;
    }

    // compute_root (utils.cu:94-135) of the leaf in `a` (lane i < NL) over the
    // auth path at auth; masks: 2 NL lanes per H (robust)
    SPX_DEV static uint64_t climb(uint64_t a, const KeccakLane &k, uint32_t lane, const uint8_t *pk, int hp, Adrs ad,
                                  uint32_t idx, const uint8_t *auth, const uint64_t *masks) {
        const int v = (int)lane - PL;   // value lane of l || r
        const bool in = v >= 0 && v < 2 * NL;
        for (int h = 0; h < hp; h++) {
            const bool right = (idx >> h) & 1u;
            adrs_height(ad, h + 1);
            adrs_index(ad, idx >> (h + 1));
            const uint64_t mine = shfl64(a, (uint32_t)(v - (right ? NL : 0)) & 31u);
            uint64_t x = lane < (uint32_t)PL ? prefix(pk, ad, lane) : 0ull;
            if (in) {
                const bool own = (v >= NL) == right;
                x = own ? mine : reinterpret_cast<const uint64_t *>(auth + (uint64_t)h * N)[right ? v : v - NL];
                if (HF::kRobust) x ^= masks[h * 2 * NL + v];
            }
            if (lane == PL + 2 * NL) x ^= 0x1Full;
            if (lane == 16) x ^= 0x8000000000000000ull;
            a = x;
            warp_keccak_f1600(a, k, lane);
        }
        return a;
    }

    // the root of layer L (-1: the FORS key): lane i < NL returns lane i;
    // masks: the layer's, see mask_lanes (robust, L >= 0)
    template <class LD>
    SPX_DEV static uint64_t layer_root(const SetParams &P, const KeccakLane &k, uint32_t lane, const uint8_t *pk,
                                       uint64_t tree, uint32_t idx_leaf, const uint8_t *auth, const uint64_t *masks,
                                       int L, LD ld) {
        uint64_t tree_L = tree;
        uint32_t idx_L = idx_leaf;
        Adrs pa;
        adrs_zero(pa);
        if (L >= 0) {
            layer_index(P, tree, idx_leaf, L, tree_L, idx_L);
            adrs_layer(pa, L);
        }
        adrs_tree(pa, tree_L);
        adrs_keypair(pa, idx_L);
        adrs_type(pa, L < 0 ? ADDR_FORSPK : ADDR_WOTSPK);
        if (L < 0) return tl(k, lane, pk, pa, P.k, true, ld);
        const uint64_t a = tl(k, lane, pk, pa, LEN, false,
                              [&](uint32_t q) { return HF::kRobust ? ld(q) ^ masks[q] : ld(q); });
        Adrs ad;
        adrs_zero(ad);
        adrs_layer(ad, L);
        adrs_tree(ad, tree_L);
        adrs_type(ad, ADDR_HASHTREE);
        return climb(a, k, lane, pk, P.hp, ad, idx_L, auth, masks + LEN * NL);
    }

    // checksum of the message in lanes i < NL (chain_lengths, wots.cu:84-166), shifted as its digits are read
    SPX_DEV static uint32_t checksum(uint64_t a, uint32_t lane) {
        const uint32_t lo = (uint32_t)a, hi = (uint32_t)(a >> 32);
        uint32_t s = __dp4a((lo & 0x0f0f0f0fu) + (lo >> 4 & 0x0f0f0f0fu), 0x01010101u, 0u);
        s = __dp4a((hi & 0x0f0f0f0fu) + (hi >> 4 & 0x0f0f0f0fu), 0x01010101u, s);
        return (15u * LEN1 - __reduce_add_sync(0xffffffffu, lane < (uint32_t)NL ? s : 0u)) << 4;
    }
    // digit c (of this lane's choice; every lane calls this)
    SPX_DEV static uint32_t digit(uint64_t a, uint32_t csum, uint32_t c) {
        const uint64_t x = shfl64(a, c < (uint32_t)LEN1 ? c >> 4 : 0u);
        if (c < (uint32_t)LEN1) return (uint32_t)(x >> (8 * (c >> 1 & 7) + (c & 1 ? 0 : 4))) & 15u;
        return csum >> (12 - 4 * (c - LEN1)) & 15u;
    }
};

// One thread's mask task of a robust SHAKE layer: part 0 squeezes T_len's mask,
// SHAKE256(PUB_SEED || ADRS_T, len n bytes), part 1 the auth path's, 2n bytes
// per H; both into out (ShakeGroup::mask_lanes).
template <class HF>
SPX_DEV void shake_mask_task(const SetParams &P, const KeyRegs<4 * HF::W> &key, uint64_t tree, uint32_t idx_leaf, int L,
                             int part, uint64_t *out) {
    using SG = ShakeGroup<HF>;
    constexpr int NL = SG::NL, Q = SG::LEN * NL;
    uint64_t tree_L;
    uint32_t idx_L;
    layer_index(P, tree, idx_leaf, L, tree_L, idx_L);
    Adrs a;
    adrs_zero(a);
    adrs_layer(a, L);
    adrs_tree(a, tree_L);
    const int n = part == 0 ? (Q + 16) / 17 : P.hp;   // permutations
    uint64_t A[25];
#pragma unroll 1
    for (int b = 0; b < n; b++) {
        if (part == 1 || b == 0) {
            if (part == 0) {
                adrs_type(a, ADDR_WOTSPK);
                adrs_keypair(a, idx_L);
            } else {
                adrs_type(a, ADDR_HASHTREE);
                adrs_height(a, b + 1);
                adrs_index(a, idx_L >> (b + 1));
            }
            uint64_t al[4];
            adrs_lanes(a, al);
#pragma unroll
            for (int i = 0; i < 25; i++) A[i] = 0;
#pragma unroll
            for (int i = 0; i < NL; i++) A[i] = HF::vlane(key.pub, i);
#pragma unroll
            for (int i = 0; i < 4; i++) A[NL + i] = al[i];
            A[SG::PL] = 0x1Full;
            A[16] ^= 0x8000000000000000ull;
        }
        keccak_f1600(A);
        if (part == 0) {
#pragma unroll
            for (int i = 0; i < 17; i++)
                if (17 * b + i < Q) out[17 * b + i] = A[i];
        } else {
#pragma unroll
            for (int i = 0; i < 2 * NL; i++) out[Q + b * 2 * NL + i] = A[i];
        }
    }
}

// ---------------------------------------------------------------------------
// Signing: T_len of a small batch's leaves and T_k, whose latency the
// signature waits for, by the same lanes (8 a value sequence for SHA-256, a
// warp for SHAKE-256).  One signature, against one thread a sequence: T_len
// 23 -> 16 us at 128f, 352 -> 85 us at 256f-robust, 100 -> 60 us at SHAKE-256f.
// ---------------------------------------------------------------------------
template <class HF>
struct TlLanes {
    static constexpr int kLanes = HF::kShake ? 32 : 8, kThreads = HF::kShake ? 128 : 32;
    static constexpr int kPerBlock = kThreads / kLanes;
    // dynamic shared memory of a block
    static constexpr size_t smem() {
        if constexpr (HF::kShake) return 0;
        else return (size_t)kPerBlock * ShaGroup<HF>::kStride * 4;
    }
    // out <- T_l of m values at vals under pa (pub: PUB_SEED in memory); every
    // thread of the block calls this, `live` ones store
    SPX_DEV static void run(uint8_t *out, bool live, const KeyRegs<4 * HF::W> &key, const uint8_t *pub, const Adrs &pa,
                            int m, const uint8_t *vals) {
        extern __shared__ __align__(16) uint32_t smem[];
        const uint32_t lane = threadIdx.x % kLanes;
        if constexpr (HF::kShake) {
            using SG = ShakeGroup<HF>;
            if (!live) return;   // uniform over the warp
            KeccakLane k;
            keccak_lane_init(k, lane);
            const uint64_t a = SG::tl(k, lane, pub, pa, m, true, [&](uint32_t q) {
                return reinterpret_cast<const uint64_t *>(vals)[q];
            });
            if (lane < (uint32_t)SG::NL) reinterpret_cast<uint64_t *>(out)[lane] = a;
        } else {
            using SG = ShaGroup<HF>;
            uint32_t v[HF::W];
            SG::template tl<kLanes>(v, smem + threadIdx.x / kLanes * SG::kStride, lane, key, pa, m, true,
                                    [&](uint32_t q) { return reinterpret_cast<const uint2 *>(vals)[q]; });
            if (live && lane == 0) HF::store(out, v);
        }
    }
};

// T_len over a leaf's chain ends, in succession (chain_end)
template <class HF>
__global__ void __launch_bounds__(TlLanes<HF>::kThreads) k_leaf_tlen(SetParams P, LeafArgs A) {
    constexpr int N = 4 * HF::W, LEN = 2 * N + 3;
    const uint32_t x0 = (blockIdx.x * blockDim.x + threadIdx.x) / TlLanes<HF>::kLanes;
    const bool live = x0 >> P.hp < A.trees;
    const uint32_t x = live ? x0 : 0;
    KeyRegs<N> key;
    Adrs pa;
    uint8_t *to;
    const uint8_t *sk = tlen_pos<HF>(P, A, x, key, pa, to);
    TlLanes<HF>::run(to, live, key, sk + 2 * N, pa, LEN, chain_end<N>(A, x, 0));
}

// T_k over a signature's FORS roots (fors.cu:141-142), in place of the first
// root.  Runs behind k_fors_sign, beside the hypertree.
template <class HF>
__global__ void __launch_bounds__(TlLanes<HF>::kThreads) k_fors_pk(SetParams P, SignArgs A) {
    constexpr int N = 4 * HF::W;
    const uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) / TlLanes<HF>::kLanes;
    const bool live = i0 < A.count;
    const uint32_t item = live ? i0 : A.count - 1;
    const SignWork &wk = A.work[item];
    const uint8_t *sk = A.sk.row(item);
    KeyRegs<N> key;
    key_from_work<HF>(key, sk, sk + 2 * N, wk);
    Adrs pa;
    adrs_zero(pa);
    adrs_tree(pa, wk.tree);
    adrs_keypair(pa, wk.idx_leaf);
    adrs_type(pa, ADDR_FORSPK);
    uint8_t *roots = A.fors_roots + (uint64_t)item * P.k * N;
    TlLanes<HF>::run(roots, live, key, sk + 2 * N, pa, P.k, roots);
}

}  // namespace cuspx
