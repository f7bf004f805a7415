// spx_vblock.cuh -- SHA-256 verify of a batch's whole hypertree in one launch.
//
// A block keeps I items.  Per layer its threads take one WOTS+ chain each,
// sorted by length within the block (a warp runs as long as its longest
// chain, so mixed lengths idle half its lanes: see spx_vsort.cuh), then warp 0
// runs T_len and the auth paths with 32 / I lanes an item (spx_vgroup.cuh)
// while the other warps fetch the next layer's signature values and auth
// paths.  Nothing leaves the block between layers, so a layer costs its
// longest chain and its serial path, without launches, bucket lists or a trip
// through memory, and one block's serial path runs beside other blocks'
// chains on the same SM.
#pragma once
#include "spx_vgroup.cuh"
#include "spx_vsort.cuh"

namespace cuspx {

template <class HF, int I>
struct VerifyBlock {
    using SG = ShaGroup<HF>;
    static constexpr int W = SG::W, N = SG::N, LEN = SG::LEN, G = 32 / I, kChains = I * LEN;
    static constexpr int kThreads = kChains <= 64 ? 64 : (kChains + 31) / 32 * 32;
    // an item's fixed data
    enum : int { T_MID = 0, T_PUB = 8, T_TREE = 16, T_LEAF = 18, T_ITEM, T_OK, T_CSUM, kInfo = 24 };
    // shared words: I ShaGroup areas, I x info, the chain ends, the sort, and
    // two buffers of the layer's signature values and auth path
    static constexpr int S_INFO = I * SG::kStride, S_VALS = S_INFO + I * kInfo, S_ORDER = S_VALS + kChains * W,
                         S_HIST = S_ORDER + (kChains + 3) / 4 * 4, S_ROWS = S_HIST + 16;
    SPX_HD static int row_words(int hp) { return (LEN + hp) * W; }
    SPX_HD static int words(int hp) { return S_ROWS + 2 * I * row_words(hp); }
};

template <class HF, int I>
__global__ void __launch_bounds__(VerifyBlock<HF, I>::kThreads) k_verify_block(SetParams P, VerifyArgs A) {
    using V = VerifyBlock<HF, I>;
    using SG = ShaGroup<HF>;
    constexpr int W = V::W, N = V::N, LEN = V::LEN, G = V::G;
    extern __shared__ __align__(16) uint32_t smem[];
    uint32_t *hist = smem + V::S_HIST, *order = smem + V::S_ORDER, *vals = smem + V::S_VALS;
    const uint32_t t = threadIdx.x;
    const uint32_t first = blockIdx.x * I;
    const int rw = V::row_words(P.hp);
    auto info = [&](uint32_t it) { return smem + V::S_INFO + it * V::kInfo; };
    auto rows = [&](int L, uint32_t it) { return smem + V::S_ROWS + ((L & 1) * I + it) * rw; };
    auto key_of = [&](KeyRegs<N> &key, uint32_t it) {
        const uint32_t *f = info(it);
#pragma unroll
        for (int i = 0; i < 8; i++) key.mid[i] = f[V::T_MID + i];
#pragma unroll
        for (int i = 0; i < W; i++) key.pub[i] = f[V::T_PUB + i];
    };
    auto tree_of = [&](uint32_t it) { return (uint64_t)info(it)[V::T_TREE + 1] << 32 | info(it)[V::T_TREE]; };
    // layer L's signature values and auth paths of the block's items (contiguous
    // in a signature), by every warp but the first
    auto fetch = [&](int L) {
        const int per = rw / 2;
        for (int e = (int)t - 32; e < I * per; e += V::kThreads - 32) {
            const int it = e / per, q = e - it * per;
            const uint8_t *src = A.sig + (uint64_t)info(it)[V::T_ITEM] * A.sig_stride + sig_layer_off(P, L);
            reinterpret_cast<uint2 *>(rows(L, it))[q] = reinterpret_cast<const uint2 *>(src)[q];
        }
    };
    if (t < I) {
        const uint32_t i = first + t;
        const bool live = i < A.count;
        const uint32_t item = live ? i : A.count - 1;   // a part-full block repeats the last item
        const SignWork &wk = A.work[item];
        uint32_t *f = info(t);
        uint32_t pub[W];
        HF::load(pub, A.pk.row(item));
#pragma unroll
        for (int x = 0; x < 8; x++) f[V::T_MID + x] = wk.mid[x];
#pragma unroll
        for (int x = 0; x < W; x++) f[V::T_PUB + x] = pub[x];
        f[V::T_TREE] = (uint32_t)wk.tree;
        f[V::T_TREE + 1] = (uint32_t)(wk.tree >> 32);
        f[V::T_LEAF] = wk.idx_leaf;
        f[V::T_ITEM] = item;
        f[V::T_OK] = !live ? 2u : (wk.flags ? 0u : 1u);   // 0: wrong signature length (sign.cu:3063-3065)
    }
    if (t < 16) hist[t] = 0;
    __syncthreads();
#pragma unroll 1
    for (int L = -1; L < P.d; L++) {
        if (L >= 0) {
            // sort the block's chains, longest first
            const uint32_t it0 = t / LEN;
            uint32_t l = 0, rank = 0;
            if (t < V::kChains) {
                l = 15u - SG::digit(smem + it0 * SG::kStride, info(it0)[V::T_CSUM], t - it0 * LEN);
                rank = atomicAdd(&hist[l], 1u);
            }
            __syncthreads();
            if (t < V::kChains) {
                for (uint32_t b = l + 1; b < 16; b++) rank += hist[b];
                order[rank] = l << 16 | t;
            }
            __syncthreads();
            if (t < 16) hist[t] = 0;
            if (t < V::kChains) {
                const uint32_t e = order[t], id = e & 0xffffu, it = id / LEN, c = id - it * LEN;
                KeyRegs<N> key;
                key_of(key, it);
                uint64_t tree_L;
                uint32_t idx_L;
                layer_index(P, tree_of(it), info(it)[V::T_LEAF], L, tree_L, idx_L);
                Adrs wa;
                adrs_zero(wa);
                adrs_layer(wa, L);
                adrs_tree(wa, tree_L);
                adrs_type(wa, ADDR_WOTS);
                adrs_keypair(wa, idx_L);
                adrs_chain(wa, c);
                uint32_t v[W];
                HF::load(v, reinterpret_cast<const uint8_t *>(rows(L, it) + c * W));
                typename HF::FCtx fc;
                HF::f_prepare(fc, wa, key);
                HF::chain_in(v);
                for (uint32_t s = 15u - (e >> 16); s < 15u; s++) HF::f_step(v, v, fc, s, key);
                HF::chain_out(v);
                tlen_mask_value<HF>(v, key, L, tree_L, idx_L, (int)c);
                HF::store(reinterpret_cast<uint8_t *>(vals + id * W), v);
            }
            __syncthreads();
        }
        if (t < 32) {
            const uint32_t it = t / G, g = t % G, item = info(it)[V::T_ITEM], ok = info(it)[V::T_OK];
            uint32_t *S = smem + it * SG::kStride;
            KeyRegs<N> key;
            key_of(key, it);
            const uint2 *src = L < 0 ? reinterpret_cast<const uint2 *>(A.fors_roots + (uint64_t)item * P.k * N)
                                     : reinterpret_cast<const uint2 *>(vals + it * LEN * W);
            uint32_t root[W];
            SG::template layer_root<G>(root, P, S, g, key, tree_of(it), info(it)[V::T_LEAF],
                                       reinterpret_cast<const uint8_t *>(rows(L < 0 ? 0 : L, it) + LEN * W), L,
                                       [&](uint32_t q) { return src[q]; });
            if (g == 0) {
                if (L == P.d - 1) {
                    if (ok != 2) {
                        uint32_t pr[W];
                        HF::load(pr, A.pk.row(item) + N);
                        bool eq = ok == 1;
#pragma unroll
                        for (int x = 0; x < W; x++) eq &= pr[x] == root[x];
                        A.verdict[item] = eq ? 0 : -1;
                    }
                } else {
#pragma unroll
                    for (int x = 0; x < W; x++) S[SG::S_ROOT + x] = root[x];
                    info(it)[V::T_CSUM] = SG::checksum(root);
                }
            }
        } else if (L + 1 < P.d) {
            fetch(L + 1);
        }
        __syncthreads();
    }
}

}  // namespace cuspx
