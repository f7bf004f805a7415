// spx_thash.cuh -- SPHINCS+ tweakable hash families on top of spx_hash.cuh.
//
// Two policy classes with one interface, instantiated per (n, robust):
//   Sha2<N, ROBUST>   thash_sha256.cu:16-34 (simple), hash_sha256.cu:65-326
//   Shake<N, ROBUST>  thash_shake256.cu:15-25 (simple), hash_shake256.cu:38-130
// Robust thash is not in the reference; it follows the published SPHINCS+
// round-3 robust construction: the input is xored with a bitmask drawn from
// MGF1-SHA256(PUB_SEED || ADRS_c) or SHAKE256(PUB_SEED || ADRS).
//
//   F(out, in, adrs, key)        one n-byte block
//   H(out, l, r, adrs, key)      two n-byte blocks
//   PRF(out, adrs, key)          secret chain/leaf start value
//   TStream                      T_l over a stream of n-byte values (T_len,
//                                T_k), absorbing as values are produced
//   prf_msg / h_msg              message randomiser and message digest over
//                                a message in global memory
#pragma once
#include "spx_hash.cuh"

#ifndef CUSPX_ROBUST_LEAF_MINBLOCKS
#define CUSPX_ROBUST_LEAF_MINBLOCKS 1
#endif

namespace cuspx {

// Per-item key material in registers.  mid is the SHA-256 state after the
// 64-byte block PUB_SEED || 0^(64-n) (the reference's process-global
// state_seeded, sha256.cu:385-405, here one per key).
template <int N>
struct KeyRegs {
    static constexpr int W = N / 4;
    uint32_t pub[W];
    uint32_t skseed[W];
    uint32_t mid[8];
};

// ---------------------------------------------------------------------------
// global-memory helpers for n-byte strings (all offsets multiples of 8)
// ---------------------------------------------------------------------------
template <int N>
SPX_DEV void load_bytes_le(uint32_t v[N / 4], const uint8_t *p) {
    if (N % 16 == 0 && ((uintptr_t)p & 15) == 0) {
#pragma unroll
        for (int i = 0; i < N / 16; i++) {
            uint4 q = reinterpret_cast<const uint4 *>(p)[i];
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < N / 8; i++) {
            uint2 q = reinterpret_cast<const uint2 *>(p)[i];
            v[2 * i] = q.x; v[2 * i + 1] = q.y;
        }
    }
}
template <int N>
SPX_DEV void store_bytes_le(uint8_t *p, const uint32_t v[N / 4]) {
    if (N % 16 == 0 && ((uintptr_t)p & 15) == 0) {
#pragma unroll
        for (int i = 0; i < N / 16; i++)
            reinterpret_cast<uint4 *>(p)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < N / 8; i++) reinterpret_cast<uint2 *>(p)[i] = make_uint2(v[2 * i], v[2 * i + 1]);
    }
}

// ===========================================================================
// SHA-256 family
// ===========================================================================
// second block of a robust n = 32 bitmask (PUB_SEED || ADRS_c || ctr, 58 bytes)
static __constant__ Sha256PadKw c_mask_pad = sha256_pad_kw(58 * 8);

template <int N, bool ROBUST>
struct Sha2 {
    static constexpr int W = N / 4;
    static constexpr bool kRobust = ROBUST;
    static constexpr int kShake = 0;
    static constexpr bool kFmaA = !ROBUST;   // the round's form, see sha256_rounds
    // k_leaves occupancy floor for robust chains (which carry a second, mask
    // state); measured on GB300, capping registers to raise it spills and is
    // slower, so the default leaves the compiler's choice
    static constexpr int kLeafMinBlocks = ROBUST ? CUSPX_ROBUST_LEAF_MINBLOCKS : 1;

    // memory <-> register order
    SPX_DEV static void load(uint32_t v[W], const uint8_t *p) {
        load_bytes_le<N>(v, p);
#pragma unroll
        for (int i = 0; i < W; i++) v[i] = bswap32(v[i]);
    }
    SPX_DEV static void store(uint8_t *p, const uint32_t v[W]) {
        uint32_t t[W];
#pragma unroll
        for (int i = 0; i < W; i++) t[i] = bswap32(v[i]);
        store_bytes_le<N>(p, t);
    }

    // midstate after PUB_SEED || 0^(64-n)  (seed_state, sha256.cu:391-405)
    SPX_DEV static void key_init(KeyRegs<N> &k, const uint8_t *skseed, const uint8_t *pub) {
        load(k.skseed, skseed);
        load(k.pub, pub);
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = i < W ? k.pub[i] : 0u;
        sha256_iv(k.mid);
        sha256_compress<kFmaA>(k.mid, w);
    }

    // ---- thash as a sequence of compressions --------------------------------
    // thash over L words is kUnits<L> compressions: robust sets first draw
    // each bitmask block (kMaskUnits of them per 8 input words), then the
    // message's blocks follow.  They run through one compression call site
    // with a loop around it: a site is 20 KB of unrolled rounds, and a kernel
    // with several on its hot path waits for instructions: FORS trees with
    // PRF, F and H each on their own kept the ALU pipe 74% (128f), 54% (192f)
    // and 57% (256f-robust) busy, with 4.6 to 6.7 cycles of `no_instruction`
    // an issue; 1024 signatures of 192f took 3.00 ms there, through one site
    // 2.10 ms, 100 of 256s-robust 34 and 22 ms.  (Rolling the rounds instead
    // is slower: 16.2 against 16.7 G compressions/s.)
    template <int L>
    static constexpr int kBlocks = (22 + 4 * L + 9 + 63) / 64;
    static constexpr int kMaskUnits = (N + 26 + 9 + 63) / 64;
    template <int L>
    static constexpr int kMaskAll = ROBUST ? (L + 7) / 8 * kMaskUnits : 0;
    template <int L>
    static constexpr int kUnits = kMaskAll<L> + kBlocks<L>;

    // block b of SHA256(midstate; ADRS_c || in[L words]) (thash_sha256.cu:16-34)
    template <int L>
    SPX_DEV static void core_block(uint32_t w[16], const Adrs &a, const uint32_t in[L], int b) {
        constexpr int NB = kBlocks<L>;
        uint32_t m[16 * NB];
#pragma unroll
        for (int i = 0; i < 5; i++) m[i] = a.w[i];
        m[5] = (a.w[5] & 0xffff0000u) | (in[0] >> 16);
#pragma unroll
        for (int i = 1; i < L; i++) m[5 + i] = __funnelshift_l(in[i], in[i - 1], 16);
        m[5 + L] = (in[L - 1] << 16) | 0x8000u;
#pragma unroll
        for (int i = 6 + L; i < 16 * NB; i++) m[i] = 0;
        m[16 * NB - 1] = (64 + 22 + 4 * L) * 8;
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = NB == 1 || b == 0 ? m[i] : m[16 * (NB - 1) + i];
    }
    // first block of MGF1-SHA256(PUB_SEED || ADRS_c, .) block `ctr` (sha256.cu:
    // 362-383), from the IV; at n = 32 the length block follows (pad_block)
    SPX_DEV static void mask_words(uint32_t w[16], const uint32_t pub[W], const Adrs &a, uint32_t ctr) {
        constexpr int TOT = N + 26;
#pragma unroll
        for (int i = 0; i < W; i++) w[i] = pub[i];
#pragma unroll
        for (int i = 0; i < 5; i++) w[W + i] = a.w[i];
        w[W + 5] = (a.w[5] & 0xffff0000u) | (ctr >> 16);
        w[W + 6] = (ctr << 16) | 0x8000u;
#pragma unroll
        for (int i = W + 7; i < 16; i++) w[i] = 0;
        if (kMaskUnits == 1) w[15] = TOT * 8;
    }
    SPX_DEV static void pad_block(uint32_t st[8]) {
        uint32_t t[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = st[i];
        sha256_rounds_pad<kFmaA>(t, c_mask_pad);
#pragma unroll
        for (int i = 0; i < 8; i++) st[i] += t[i];
    }
    SPX_DEV static void mask_block(uint32_t out[8], const uint32_t pub[W], const Adrs &a, uint32_t ctr) {
        uint32_t w[16];
        mask_words(w, pub, a, ctr);
        sha256_iv(out);
        sha256_compress<kFmaA>(out, w);
        if (kMaskUnits == 2) pad_block(out);
    }
    // unit u of thash over in is the length block of a bitmask
    template <int L>
    SPX_DEV static bool pad_unit(int u) {
        return ROBUST && kMaskUnits == 2 && u < kMaskAll<L> && u % 2 == 1;
    }
    // block words w and start state st of any other unit (st holds the unit
    // before's result where the unit continues it), ...
    template <int L>
    SPX_DEV static void unit_block(uint32_t w[16], uint32_t st[8], const KeyRegs<N> &k, const Adrs &a,
                                   const uint32_t in[L], int u) {
        constexpr int MU = kMaskAll<L>;
        if (ROBUST && u < MU) {
            sha256_iv(st);
            mask_words(w, k.pub, a, (uint32_t)(u / kMaskUnits));
        } else {
            if (u == MU) {
#pragma unroll
                for (int i = 0; i < 8; i++) st[i] = k.mid[i];
            }
            core_block<L>(w, a, in, u - MU);
        }
    }
    // ... and what follows its compression: a finished bitmask block goes into in
    template <int L>
    SPX_DEV static void unit_done(const uint32_t st[8], uint32_t in[L], int u) {
        if (ROBUST && u < kMaskAll<L> && u % kMaskUnits == kMaskUnits - 1) {
#pragma unroll
            for (int b = 0; b < (L + 7) / 8; b++)
                if (b == u / kMaskUnits) {
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        if (8 * b + i < L) in[8 * b + i] ^= st[i];
                }
        }
    }
    template <int L>
    SPX_DEV static void thash(uint32_t out[W], const KeyRegs<N> &k, const Adrs &a, uint32_t in[L]) {
        uint32_t st[8];
#pragma unroll
        for (int i = 0; i < 8; i++) st[i] = k.mid[i];
#pragma unroll 1
        for (int u = 0; u < kUnits<L>; u++) {
            if (pad_unit<L>(u)) {
                pad_block(st);
            } else {
                uint32_t w[16];
                unit_block<L>(w, st, k, a, in, u);
                sha256_compress<kFmaA>(st, w);
            }
            unit_done<L>(st, in, u);
        }
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = st[i];
    }

    SPX_DEV static void F(uint32_t out[W], const uint32_t in[W], const Adrs &a, const KeyRegs<N> &k) {
        uint32_t t[W];
#pragma unroll
        for (int i = 0; i < W; i++) t[i] = in[i];
        thash<W>(out, k, a, t);
    }
    SPX_DEV static void H(uint32_t out[W], const uint32_t l[W], const uint32_t r[W], const Adrs &a,
                          const KeyRegs<N> &k) {
        uint32_t t[2 * W];
#pragma unroll
        for (int i = 0; i < W; i++) { t[i] = l[i]; t[W + i] = r[i]; }
        thash<2 * W>(out, k, a, t);
    }

    // ---- WOTS+ chain steps ------------------------------------------------
    // Along one chain the ADRS differs only in its hash byte (byte 21, in
    // message word 5), so rounds 0..4 of every F compression -- and rounds
    // 0..W+4 of the robust mask compression -- are the same for all steps.
    // f_prepare runs them once; f_step starts each compression after them.
    struct FCtx {
        uint32_t st[8];     // state after rounds 0..4 from the midstate
        uint32_t m[5];      // ADRS words 0..4
        uint32_t a5;        // ADRS word 5 without the hash byte
        uint32_t mst[ROBUST ? 8 : 1];   // robust: mask state after rounds 0..W+4 from the IV
    };
    SPX_DEV static void f_prepare(FCtx &f, const Adrs &a, const KeyRegs<N> &k) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 5; i++) f.m[i] = w[i] = a.w[i];
        f.a5 = a.w[5] & 0xff000000u;
#pragma unroll
        for (int i = 0; i < 8; i++) f.st[i] = k.mid[i];
        sha256_rounds<0, 5, kFmaA>(f.st, w);
        if (ROBUST) {
            uint32_t x[16];
#pragma unroll
            for (int i = 0; i < W; i++) x[i] = k.pub[i];
#pragma unroll
            for (int i = 0; i < 5; i++) x[W + i] = a.w[i];
            sha256_iv(f.mst);
            sha256_rounds<0, W + 5, kFmaA>(f.mst, x);
        }
    }
    // a chain's value needs no form of its own here (see Shake)
    SPX_DEV static void chain_in(uint32_t *) {}
    SPX_DEV static void chain_out(uint32_t *) {}
    SPX_DEV static void chain_store(uint8_t *p, const uint32_t v[W]) { store(p, v); }
    // out = F(in) at hash address `hash` of the prepared chain
    SPX_DEV static void f_step(uint32_t out[W], const uint32_t in[W], const FCtx &f, uint32_t hash,
                               const KeyRegs<N> &k) {
        const uint32_t a5 = f.a5 | (hash << 16);
        uint32_t x[W];
#pragma unroll
        for (int i = 0; i < W; i++) x[i] = in[i];
        if (ROBUST) {
            // bitmask block 0 = SHA256(PUB_SEED || ADRS_c || BE32(0)), resumed after the prefix
            constexpr int TOT = N + 26;
            constexpr int NB = (TOT + 9 + 63) / 64;
            uint32_t mw[16 * NB];
#pragma unroll
            for (int i = 0; i < W; i++) mw[i] = k.pub[i];
#pragma unroll
            for (int i = 0; i < 5; i++) mw[W + i] = f.m[i];
            mw[W + 5] = a5;
            mw[W + 6] = 0x8000u;
#pragma unroll
            for (int i = W + 7; i < 16 * NB; i++) mw[i] = 0;
            mw[16 * NB - 1] = TOT * 8;
            uint32_t t[8], ms[8];
#pragma unroll
            for (int i = 0; i < 8; i++) t[i] = f.mst[i];
            sha256_rounds<W + 5, 64, kFmaA>(t, mw);
#pragma unroll
            for (int i = 0; i < 8; i++) ms[i] = t[i] + sha256_iv_word(i);
            if (NB == 2) pad_block(ms);
#pragma unroll
            for (int i = 0; i < W; i++) x[i] ^= ms[i];
        }
        constexpr int TOT = 22 + N;   // always one block for n <= 32
        uint32_t m[16];
#pragma unroll
        for (int i = 0; i < 5; i++) m[i] = f.m[i];
        m[5] = a5 | (x[0] >> 16);
#pragma unroll
        for (int i = 1; i < W; i++) m[5 + i] = __funnelshift_l(x[i], x[i - 1], 16);
        m[5 + W] = (x[W - 1] << 16) | 0x8000u;
#pragma unroll
        for (int i = 6 + W; i < 16; i++) m[i] = 0;
        m[15] = (64 + TOT) * 8;
        uint32_t t[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = f.st[i];
        sha256_rounds<5, 64, kFmaA>(t, m);
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = t[i] + k.mid[i];
    }

    // PRF = SHA256(SK_SEED || ADRS_c), no midstate (hash_sha256.cu:65-77)
    SPX_DEV static void prf_words(uint32_t m[16], const Adrs &a, const KeyRegs<N> &k) {
#pragma unroll
        for (int i = 0; i < W; i++) m[i] = k.skseed[i];
#pragma unroll
        for (int i = 0; i < 5; i++) m[W + i] = a.w[i];
        m[W + 5] = (a.w[5] & 0xffff0000u) | 0x8000u;
#pragma unroll
        for (int i = W + 6; i < 16; i++) m[i] = 0;
        m[15] = (N + 22) * 8;
    }
    SPX_DEV static void PRF(uint32_t out[W], const Adrs &a, const KeyRegs<N> &k) {
        uint32_t m[16], s[8];
        prf_words(m, a, k);
        sha256_iv(s);
        sha256_compress<kFmaA>(s, m);
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = s[i];
    }

    // Root v of a FORS subtree of 2^sub leaves from leaf j0 (of the tree at
    // leaf offset off), by one thread with a stack of sub + 1 values
    // (treehash, utils.cu:189-241): a leaf's PRF and F and the merges it
    // completes, every compression of them through one call site (see thash).
    // sec(j, x) sees each leaf's secret, node(h, i, x) each node i of height h.
    template <class S, class T>
    SPX_DEV static void fors_subtree(uint32_t v[W], Adrs &ad, const KeyRegs<N> &k, uint32_t j0, int sub, uint32_t off,
                                     uint32_t *stk, S sec, T node) {
        uint32_t jj = 0, x[2 * W], st[8];
        int hgt = -1, u = 0;   // hgt: height of the node in the making, -1 a leaf's secret
#pragma unroll
        for (int i = 0; i < 2 * W; i++) x[i] = 0;
        adrs_height(ad, 0);
        adrs_index(ad, off + j0);
#pragma unroll 1
        for (;;) {
            if ((hgt == 0 && pad_unit<W>(u)) || (hgt > 0 && pad_unit<2 * W>(u))) {
                pad_block(st);
            } else {
                uint32_t w[16];
                if (hgt < 0) {
                    prf_words(w, ad, k);
                    sha256_iv(st);
                } else if (hgt == 0) {
                    unit_block<W>(w, st, k, ad, x, u);
                } else {
                    unit_block<2 * W>(w, st, k, ad, x, u);
                }
                sha256_compress<kFmaA>(st, w);
            }
            if (hgt < 0) {
#pragma unroll
                for (int i = 0; i < W; i++) x[i] = st[i];
                sec(j0 + jj, x);
                hgt = u = 0;
                continue;
            }
            if (hgt == 0) unit_done<W>(st, x, u);
            else unit_done<2 * W>(st, x, u);
            if (++u < (hgt == 0 ? kUnits<W> : kUnits<2 * W>)) continue;
            u = 0;
            // st: node (j0 + jj) >> hgt of height hgt
            node(hgt, (j0 + jj) >> hgt, st);
            if ((jj >> hgt) & 1u) {   // a right child: merge with the stack's top
                const uint32_t *top = stk + (__popc(jj >> hgt) - 1) * W;
#pragma unroll
                for (int i = 0; i < W; i++) {
                    x[i] = top[i];
                    x[W + i] = st[i];
                }
                hgt++;
                adrs_height(ad, hgt);
                adrs_index(ad, ((j0 + jj) >> hgt) + (off >> hgt));
                continue;
            }
            if (jj + 1 == 1u << sub) break;
            // a left child waits on the stack, above an entry per set bit
            uint32_t *top = stk + __popc(jj >> hgt) * W;
#pragma unroll
            for (int i = 0; i < W; i++) top[i] = st[i];
            jj++;
            hgt = -1;
            adrs_height(ad, 0);
            adrs_index(ad, off + j0 + jj);
        }
#pragma unroll
        for (int i = 0; i < W; i++) v[i] = st[i];
    }

    // T_l streaming: midstate; ADRS_c || v_0 || v_1 ... Every value lands at a
    // byte offset that is 2 mod 4, so each word straddles two buffer words.
    // buf is a per-thread shared-memory area of kSmemWords words.
    static constexpr int kSmemWords = 17 + (ROBUST ? 8 : 0);
    struct TStream {
        uint32_t st[8];
        uint32_t *buf;
        int pos;        // byte position in the current block, == 2 mod 4
        uint32_t q;     // data words absorbed (for the robust mask)
        uint32_t blocks;
        Adrs a;
    };
    SPX_DEV static void t_init(TStream &t, uint32_t *smem, const KeyRegs<N> &k, const Adrs &a) {
        t.buf = smem;
#pragma unroll
        for (int i = 0; i < 8; i++) t.st[i] = k.mid[i];
#pragma unroll
        for (int i = 0; i < 5; i++) t.buf[i] = a.w[i];
        t.buf[5] = a.w[5] & 0xffff0000u;
        t.pos = 22;
        t.q = 0;
        t.blocks = 0;
        t.a = a;
    }
    SPX_DEV static void t_flush(TStream &t) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = t.buf[i];
        sha256_compress<kFmaA>(t.st, w);
        t.blocks++;
    }
    SPX_DEV static void t_word(TStream &t, uint32_t x, const KeyRegs<N> &k) {
        if (ROBUST) {
            uint32_t *mb = t.buf + 17;
            if ((t.q & 7) == 0) {
                uint32_t mk[8];
                mask_block(mk, k.pub, t.a, t.q >> 3);
#pragma unroll
                for (int i = 0; i < 8; i++) mb[i] = mk[i];
            }
            x ^= mb[t.q & 7];
        }
        t.q++;
        int wi = t.pos >> 2;
        t.buf[wi] |= x >> 16;
        t.buf[wi + 1] = x << 16;
        t.pos += 4;
        if (t.pos > 64) {
            t_flush(t);
            t.buf[0] = t.buf[16];
            t.pos -= 64;
        }
    }
    SPX_DEV static void t_absorb(TStream &t, const uint32_t v[W], const KeyRegs<N> &k) {
#pragma unroll
        for (int i = 0; i < W; i++) t_word(t, v[i], k);
    }
    SPX_DEV static void t_final(uint32_t out[W], TStream &t) {
        uint32_t bits = (uint32_t)(64 + 64 * t.blocks + t.pos) * 8u;
        int wi = t.pos >> 2;
        t.buf[wi] |= 0x8000u;
        for (int i = wi + 1; i < 16; i++) t.buf[i] = 0;
        if (t.pos + 1 > 56) {
            t_flush(t);
            for (int i = 0; i < 16; i++) t.buf[i] = 0;
        }
        t.buf[15] = bits;
        t_flush(t);
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = t.st[i];
    }

    // T_l of M n-byte values: midstate; ADRS_c || values, block by block.
    // ld(q) gives bytes 8q .. 8q + 7 of the values (memory order).  A value
    // word straddles two stream words (the values start at byte 22), so block
    // j needs value words 16j - 6 .. 16j + 10; a robust set's mask block b
    // covers value words 8b .. 8b + 7.
    template <int M, class LD>
    SPX_DEV static void t_values(uint32_t out[W], const KeyRegs<N> &k, const Adrs &a, LD ld) {
        constexpr int NB = (22 + M * N + 9 + 63) / 64, Q = M * N / 8, MB = (M * N + 31) / 32;
        uint32_t st[8], mk[24];
#pragma unroll
        for (int i = 0; i < 24; i++) mk[i] = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) st[i] = k.mid[i];
#pragma unroll 1
        for (int j = 0; j < NB; j++) {
            uint32_t v[18], w[16];   // v[i]: value word 16j - 6 + i
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const int q = 8 * j - 3 + i;
                uint2 x = make_uint2(0u, 0u);
                if (q >= 0 && q < Q) x = ld((uint32_t)q);
                v[2 * i] = bswap32(x.x);
                v[2 * i + 1] = bswap32(x.y);
            }
            if constexpr (ROBUST) {
                // mk: mask blocks 2j - 1 (kept from the last block), 2j, 2j + 1
#pragma unroll 1
                for (int h = 0; h < 2; h++) {
                    uint32_t x[8];
                    mask_block(x, k.pub, a, 2 * j + h);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (h == 0) mk[8 + i] = x[i];
                        else mk[16 + i] = x[i];
                    }
                    if (2 * j + 1 >= MB) break;
                }
#pragma unroll
                for (int i = 0; i < 18; i++) {
                    const int x = 16 * j - 6 + i;
                    if (x >= 0 && x < M * W) v[i] ^= mk[2 + i];
                }
#pragma unroll
                for (int i = 0; i < 8; i++) mk[i] = mk[16 + i];
            }
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = __funnelshift_l(v[i + 1], v[i], 16);
            if (j == 0) {
#pragma unroll
                for (int i = 0; i < 5; i++) w[i] = a.w[i];
                w[5] |= a.w[5] & 0xffff0000u;
            }
            if (j == (5 + M * W) / 16) w[(5 + M * W) % 16] |= 0x8000u;
            if (j == NB - 1) w[15] = (uint32_t)(64 + 22 + M * N) * 8u;
            sha256_compress<kFmaA>(st, w);
        }
#pragma unroll
        for (int i = 0; i < W; i++) out[i] = st[i];
    }

    // ---- message hashing over a message in global memory -----------------
    // word q (big-endian) of the padded stream "prefix(P words) || m || 0x80
    // || 0* || bitlen64"; m must be 4-byte aligned and readable up to the
    // next multiple of 4 bytes.
    SPX_DEV static uint32_t msg_word(const uint8_t *m, uint64_t mlen, uint64_t q) {
        uint64_t b = 4 * q;
        if (b + 4 <= mlen) return bswap32(*reinterpret_cast<const uint32_t *>(m + b));
        if (b > mlen) return 0;
        uint32_t keep = (uint32_t)(mlen - b);  // 0..3 message bytes in this word
        uint32_t x = keep ? bswap32(*reinterpret_cast<const uint32_t *>(m + b)) : 0u;
        uint32_t hi = keep ? (0xffffffffu << (32 - 8 * keep)) : 0u;
        return (x & hi) | (0x80u << (24 - 8 * keep));
    }
    // 16 big-endian message words starting at word q0, all inside m; the
    // word offset keeps the alignment the prefix length gives (P % 4 == 0:
    // 16-byte, P even: 8-byte, else 4-byte) since m itself is 16-byte aligned
    template <int P>
    SPX_DEV static void msg_block_full(uint32_t w[16], const uint8_t *m, uint64_t q0) {
        const uint8_t *p = m + 4 * q0;
        if (P % 4 == 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 v = reinterpret_cast<const uint4 *>(p)[i];
                w[4 * i] = bswap32(v.x); w[4 * i + 1] = bswap32(v.y);
                w[4 * i + 2] = bswap32(v.z); w[4 * i + 3] = bswap32(v.w);
            }
        } else if (P % 2 == 0) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint2 v = reinterpret_cast<const uint2 *>(p)[i];
                w[2 * i] = bswap32(v.x); w[2 * i + 1] = bswap32(v.y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++) w[i] = bswap32(reinterpret_cast<const uint32_t *>(p)[i]);
        }
    }
    // Block b of prefix (P words, registers) || m || SHA-256 padding, where
    // bits is the total message length in bits.  Blocks wholly inside the
    // message come from the one-block-ahead vector load in nxt (have), and
    // block b + 1 is loaded into nxt here when it is such a block.
    template <int P>
    SPX_DEV static void next_block(uint32_t w[16], uint64_t b, uint64_t nblocks, uint64_t bits, const uint32_t pre[P],
                                   const uint8_t *m, uint64_t mlen, uint32_t nxt[16], bool &have) {
        constexpr int PB = (P + 15) / 16;  // blocks that contain prefix words
        auto full = [&](uint64_t x) { return x >= (uint64_t)PB && 4 * (16 * x - P + 16) <= mlen; };
        if (have) {
#pragma unroll
            for (int j = 0; j < 16; j++) w[j] = nxt[j];
        } else if (b < PB) {
#pragma unroll
            for (int pb = 0; pb < PB; pb++) {
                if (pb == (int)b) {
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const int g = 16 * pb + j;
                        w[j] = g < P ? pre[g < P ? g : 0] : msg_word(m, mlen, (uint64_t)(g - P));
                    }
                }
            }
        } else {
            const uint64_t q0 = 16 * b - P;
#pragma unroll
            for (int j = 0; j < 16; j++) w[j] = msg_word(m, mlen, q0 + j);
        }
        have = b + 1 < nblocks && full(b + 1);
        if (have) msg_block_full<P>(nxt, m, 16 * (b + 1) - P);
        if (b == nblocks - 1) {
            w[14] = (uint32_t)(bits >> 32);
            w[15] = (uint32_t)bits;
        }
    }

    // absorb prefix (P words, registers) || m into st, which has already
    // absorbed pre_blocks 64-byte blocks; out = final state.
    template <int P>
    SPX_DEV static void stream_msg(uint32_t st[8], uint32_t pre_blocks, const uint32_t pre[P], const uint8_t *m,
                                   uint64_t mlen) {
        const uint64_t dbytes = 4 * (uint64_t)P + mlen;
        const uint64_t nblocks = (dbytes + 9 + 63) / 64;
        const uint64_t bits = (64 * (uint64_t)pre_blocks + dbytes) * 8;
        uint32_t nxt[16];
        bool have = false;
        for (uint64_t b = 0; b < nblocks; b++) {
            uint32_t w[16];
            next_block<P>(w, b, nblocks, bits, pre, m, mlen, nxt, have);
            sha256_compress<kFmaA>(st, w);
        }
    }

    // The same absorption split over the two warps of a 64-thread block that
    // hashes 32 messages, for long messages: a thread hashing alone is bound
    // by its own instruction issue, about 1.3k ALU instructions per block.
    // For message l, lane l of warp 0 (role 0) builds each block and its
    // schedule with the round constants added into kw, and lane l of warp 1
    // (role 1) runs the 64 rounds from kw two blocks behind; one __syncthreads
    // hands two blocks over (one at a time: 3% slower).  kw is a shared double buffer of kPairBlocks
    // blocks x 64 words with the 32 messages interleaved (word t of buffer q
    // at kw[(q * 64 + t) * 32 + l]).
    // Every thread of the block calls this; max_blocks (the same for the
    // whole block) bounds the loop, and threads whose message has fewer
    // blocks, or role 2, only take part in the barriers.  The result is in
    // role 1's st.
    static constexpr int kPairBlocks = 2, kPairWords = 2 * kPairBlocks * 64 * 32;
    template <int P>
    SPX_DEV static void stream_msg_pair(uint32_t st[8], uint32_t pre_blocks, const uint32_t pre[P],
                                        const uint8_t *m, uint64_t mlen, uint32_t *kw, int role,
                                        uint64_t max_blocks) {
        const uint64_t dbytes = 4 * (uint64_t)P + mlen;
        const uint64_t nblocks = (dbytes + 9 + 63) / 64;
        const uint64_t bits = (64 * (uint64_t)pre_blocks + dbytes) * 8;
        uint32_t *mine = kw + (threadIdx.x & 31);
        uint32_t nxt[16];
        bool have = false;
        for (uint64_t q = 0; q <= (max_blocks + kPairBlocks - 1) / kPairBlocks; q++) {
#pragma unroll 1
            for (int u = 0; u < kPairBlocks; u++) {
                const uint64_t b = q * kPairBlocks + u;   // role 1's block is kPairBlocks earlier
                if (role == 0 && b < nblocks) {
                    uint32_t w[16];
                    next_block<P>(w, b, nblocks, bits, pre, m, mlen, nxt, have);
                    sha256_schedule_kw<32>(mine + 64 * 32 * ((q & 1) * kPairBlocks + u), w);
                }
                if (role == 1 && q > 0 && b - kPairBlocks < nblocks)
                    sha256_compress_kw<32>(st, mine + 64 * 32 * ((~q & 1) * kPairBlocks + u));
            }
            __syncthreads();
        }
    }
    // blocks of prefix (P words) || m with SHA-256 padding
    template <int P>
    SPX_DEV static uint64_t msg_blocks(uint64_t mlen) { return (4 * (uint64_t)P + mlen + 9 + 63) / 64; }

    // PRF_msg = HMAC-SHA256(SK_PRF, optrand || m), truncated (hash_sha256.cu:99-145):
    // the inner hash starts from the key block xor ipad, the outer one hashes
    // the key block xor opad and the inner digest
    SPX_DEV static void hmac_start(uint32_t st[8], const uint32_t skprf[W]) {
        uint32_t w[16];
        sha256_iv(st);
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = (i < W ? skprf[i] : 0u) ^ 0x36363636u;
        sha256_compress<kFmaA>(st, w);
    }
    SPX_DEV static void hmac_finish(uint32_t R[W], const uint32_t inner[8], const uint32_t skprf[W]) {
        uint32_t st[8], w[16];
        sha256_iv(st);
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = (i < W ? skprf[i] : 0u) ^ 0x5c5c5c5cu;
        sha256_compress<kFmaA>(st, w);
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = inner[i];
        w[8] = 0x80000000u;
#pragma unroll
        for (int i = 9; i < 15; i++) w[i] = 0;
        w[15] = (64 + 32) * 8;
        sha256_compress<kFmaA>(st, w);
#pragma unroll
        for (int i = 0; i < W; i++) R[i] = st[i];
    }
    SPX_DEV static void prf_msg(uint32_t R[W], const uint32_t skprf[W], const uint32_t optrand[W],
                                const uint8_t *m, uint64_t mlen) {
        uint32_t st[8];
        hmac_start(st, skprf);
        stream_msg<W>(st, 1, optrand, m, mlen);
        hmac_finish(R, st, skprf);
    }

    // PRF_msg (when with_prf; otherwise R is given) and H_msg of one message
    // through a single compression call site: the HMAC ipad block, optrand
    // || m, the opad block, the inner digest, R || PK || m and the MGF1
    // counter blocks run as one sequence of blocks.  With a call site per
    // step (prf_msg + h_msg) a thread hashing alone on its SM runs a fresh
    // ~20 KB copy of the unrolled rounds at every step and waits on
    // instruction fetch; here one copy stays in the instruction cache.
    // dg: dgst_bytes digest bytes (a byte array in registers/local).
    SPX_DEV static void msg_digests(uint32_t R[W], bool with_prf, const uint32_t skprf[W],
                                    const uint32_t optrand[W], const uint32_t pk[2 * W], const uint8_t *m,
                                    uint64_t mlen, uint8_t *dg, int dgst_bytes) {
        const uint64_t nb1 = (4ull * W + mlen + 9 + 63) / 64;   // optrand || m, after the ipad block
        const uint64_t bits1 = (64 + 4ull * W + mlen) * 8;
        const uint64_t nb2 = (12ull * W + mlen + 9 + 63) / 64;  // R || PK || m
        const uint64_t bits2 = (12ull * W + mlen) * 8;
        const uint64_t nm = (uint64_t)(dgst_bytes + 31) / 32;   // MGF1 blocks
        uint32_t st[8], keep[8], pre[3 * W], nxt[16];
        bool have = false;
        int phase = with_prf ? 0 : 4;   // 0 ipad, 1 optrand || m, 2 opad, 3 inner digest, 4 R || PK || m, 5 MGF1
        uint64_t b = 0;
#pragma unroll
        for (int i = 0; i < W; i++) {
            pre[i] = with_prf ? 0u : R[i];   // with_prf: R comes from phase 3
            pre[W + i] = pk[i];
            pre[2 * W + i] = pk[W + i];
        }
        sha256_iv(st);
        for (;;) {
            uint32_t w[16];
            if (phase == 0 || phase == 2) {
                const uint32_t pad = phase == 0 ? 0x36363636u : 0x5c5c5c5cu;
#pragma unroll
                for (int i = 0; i < 16; i++) w[i] = (i < W ? skprf[i] : 0u) ^ pad;
            } else if (phase == 1) {
                next_block<W>(w, b, nb1, bits1, optrand, m, mlen, nxt, have);
            } else if (phase == 4) {
                next_block<3 * W>(w, b, nb2, bits2, pre, m, mlen, nxt, have);
            } else {
                // 3: inner digest || padding (64 + 32 bytes); 5: seed || BE32(b) || padding (36 bytes)
#pragma unroll
                for (int i = 0; i < 8; i++) w[i] = keep[i];
                w[8] = phase == 3 ? 0x80000000u : (uint32_t)b;
                w[9] = phase == 3 ? 0u : 0x80000000u;
#pragma unroll
                for (int i = 10; i < 15; i++) w[i] = 0;
                w[15] = phase == 3 ? (64 + 32) * 8 : 36 * 8;
            }
            sha256_compress<kFmaA>(st, w);
            if (phase == 0) {
                phase = 1;
                b = 0;
                have = false;
            } else if (phase == 1) {
                if (++b == nb1) {
#pragma unroll
                    for (int i = 0; i < 8; i++) keep[i] = st[i];
                    sha256_iv(st);
                    phase = 2;
                }
            } else if (phase == 2) {
                phase = 3;
            } else if (phase == 3) {
#pragma unroll
                for (int i = 0; i < W; i++) R[i] = pre[i] = st[i];
                sha256_iv(st);
                phase = 4;
                b = 0;
                have = false;
            } else if (phase == 4) {
                if (++b == nb2) {
#pragma unroll
                    for (int i = 0; i < 8; i++) keep[i] = st[i];
                    sha256_iv(st);
                    phase = 5;
                    b = 0;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++)
                    if (32 * (int)b + i < dgst_bytes) dg[32 * b + i] = (uint8_t)(st[i >> 2] >> (24 - 8 * (i & 3)));
                sha256_iv(st);
                if (++b == nm) break;
            }
        }
    }

    // H_msg = MGF1-SHA256(SHA256(R || PK || m), dgst) (hash_sha256.cu:200-262);
    // writes dgst_bytes bytes to dg (a byte array in registers/local).
    SPX_DEV static void mgf1_digest(uint8_t *dg, int dgst_bytes, const uint32_t seed[8]) {
        for (int c = 0; 32 * c < dgst_bytes; c++) {
            uint32_t w[16], s[8];
#pragma unroll
            for (int i = 0; i < 8; i++) w[i] = seed[i];
            w[8] = (uint32_t)c;
            w[9] = 0x80000000u;
#pragma unroll
            for (int i = 10; i < 15; i++) w[i] = 0;
            w[15] = 36 * 8;
            sha256_iv(s);
            sha256_compress<kFmaA>(s, w);
            for (int i = 0; i < 32 && 32 * c + i < dgst_bytes; i++)
                dg[32 * c + i] = (uint8_t)(s[i >> 2] >> (24 - 8 * (i & 3)));
        }
    }
    SPX_DEV static void h_msg(uint8_t *dg, int dgst_bytes, const uint32_t R[W], const uint32_t pk[2 * W],
                              const uint8_t *m, uint64_t mlen) {
        uint32_t pre[3 * W];
#pragma unroll
        for (int i = 0; i < W; i++) pre[i] = R[i];
#pragma unroll
        for (int i = 0; i < 2 * W; i++) pre[W + i] = pk[i];
        uint32_t seed[8];
        sha256_iv(seed);
        stream_msg<3 * W>(seed, 0, pre, m, mlen);
        mgf1_digest(dg, dgst_bytes, seed);
    }
};

// ===========================================================================
// SHAKE-256 family (rate 136 bytes = 17 lanes, domain padding 0x1F..0x80)
// ===========================================================================
template <int N, bool ROBUST>
struct Shake {
    static constexpr int W = N / 4;
    static constexpr int NL = N / 8;  // lanes per value
    static constexpr bool kRobust = ROBUST;
    static constexpr int kShake = 1;
    static constexpr int kLeafMinBlocks = 1;

    SPX_DEV static void load(uint32_t v[W], const uint8_t *p) { load_bytes_le<N>(v, p); }
    SPX_DEV static void store(uint8_t *p, const uint32_t v[W]) { store_bytes_le<N>(p, v); }

    SPX_DEV static void key_init(KeyRegs<N> &k, const uint8_t *skseed, const uint8_t *pub) {
        load(k.skseed, skseed);
        load(k.pub, pub);
#pragma unroll
        for (int i = 0; i < 8; i++) k.mid[i] = 0;
    }

    SPX_DEV static uint64_t vlane(const uint32_t v[], int i) { return lane_of(v[2 * i], v[2 * i + 1]); }

    // SHAKE256(prefix(NL lanes) || ADRS(4 lanes) || in(L lanes)) -> NO lanes,
    // single permutation (every short input here is < 136 bytes)
    template <int L, int NO>
    SPX_DEV static void short_hash(uint64_t out[NO], const uint32_t pre[W], const Adrs &a, const uint64_t *in) {
        static_assert(8 * (NL + 4 + L) < 136, "short input must fit one block");
        uint64_t A[25];
        uint64_t al[4];
        adrs_lanes(a, al);
#pragma unroll
        for (int i = 0; i < 25; i++) A[i] = 0;
#pragma unroll
        for (int i = 0; i < NL; i++) A[i] = vlane(pre, i);
#pragma unroll
        for (int i = 0; i < 4; i++) A[NL + i] = al[i];
#pragma unroll
        for (int i = 0; i < L; i++) A[NL + 4 + i] = in[i];
        A[NL + 4 + L] = 0x1Full;
        A[16] ^= 0x8000000000000000ull;
        keccak_f1600_short(A);
#pragma unroll
        for (int i = 0; i < NO; i++) out[i] = A[i];
    }

    template <int L>
    SPX_DEV static void thash(uint32_t out[W], const KeyRegs<N> &k, const Adrs &a, const uint32_t in[2 * L]) {
        uint64_t x[L];
#pragma unroll
        for (int i = 0; i < L; i++) x[i] = vlane(in, i);
        if (ROBUST) {
            uint64_t mk[L];
            short_hash<0, L>(mk, k.pub, a, x);
#pragma unroll
            for (int i = 0; i < L; i++) x[i] ^= mk[i];
        }
        uint64_t o[NL];
        short_hash<L, NL>(o, k.pub, a, x);
#pragma unroll
        for (int i = 0; i < NL; i++) { out[2 * i] = (uint32_t)o[i]; out[2 * i + 1] = (uint32_t)(o[i] >> 32); }
    }

    SPX_DEV static void F(uint32_t out[W], const uint32_t in[W], const Adrs &a, const KeyRegs<N> &k) {
        thash<NL>(out, k, a, in);
    }
    SPX_DEV static void H(uint32_t out[W], const uint32_t l[W], const uint32_t r[W], const Adrs &a,
                          const KeyRegs<N> &k) {
        uint32_t t[2 * W];
#pragma unroll
        for (int i = 0; i < W; i++) { t[i] = l[i]; t[W + i] = r[i]; }
        thash<2 * NL>(out, k, a, t);
    }
    // WOTS+ chain steps, on bit-interleaved lanes (keccak_f1600_short_il):
    // the chain's value is interleaved by chain_in before the first step and
    // back by chain_out (or chain_store) after the last; the prepared chain is
    // its PUB_SEED and ADRS lanes.  (1024 signatures of SHAKE-256f: chains
    // 62.2 -> 60.9 ms.)
    struct FCtx {
        uint64_t pre[NL], ad[3];   // ad[2] without the hash byte
    };
    SPX_DEV static void f_prepare(FCtx &f, const Adrs &a, const KeyRegs<N> &k) {
        Adrs b = a;
        adrs_hash(b, 0);
        uint64_t al[4];
        adrs_lanes(b, al);
#pragma unroll
        for (int i = 0; i < NL; i++) f.pre[i] = interleave(vlane(k.pub, i));
#pragma unroll
        for (int i = 0; i < 3; i++) f.ad[i] = interleave(al[i]);
    }
    SPX_DEV static void chain_in(uint32_t v[W]) {
#pragma unroll
        for (int i = 0; i < NL; i++) {
            const uint64_t x = interleave(vlane(v, i));
            v[2 * i] = (uint32_t)x;
            v[2 * i + 1] = (uint32_t)(x >> 32);
        }
    }
    SPX_DEV static void chain_out(uint32_t v[W]) {
#pragma unroll
        for (int i = 0; i < NL; i++) {
            const uint64_t x = deinterleave(vlane(v, i));
            v[2 * i] = (uint32_t)x;
            v[2 * i + 1] = (uint32_t)(x >> 32);
        }
    }
    SPX_DEV static void chain_store(uint8_t *p, const uint32_t v[W]) {
        uint32_t t[W];
#pragma unroll
        for (int i = 0; i < W; i++) t[i] = v[i];
        chain_out(t);
        store(p, t);
    }
    SPX_DEV static void f_step(uint32_t out[W], const uint32_t in[W], const FCtx &f, uint32_t hash,
                               const KeyRegs<N> &) {
        // hash byte: ADRS byte 21, bits 40..43 of lane 2
        const uint64_t ad2 = f.ad[2] | (uint64_t)((hash >> 1 & 1u) | (hash >> 2 & 2u)) << 52 |
                             (uint64_t)((hash & 1u) | (hash >> 1 & 2u)) << 20;
        uint64_t mk[NL], A[25];
#pragma unroll
        for (int i = 0; i < NL; i++) mk[i] = 0;
#pragma unroll
        for (int pass = ROBUST ? 0 : 1; pass < 2; pass++) {   // robust: the bitmask, then F
#pragma unroll
            for (int i = 0; i < 25; i++) A[i] = 0;
#pragma unroll
            for (int i = 0; i < NL; i++) A[i] = f.pre[i];
            A[NL] = f.ad[0];
            A[NL + 1] = f.ad[1];
            A[NL + 2] = ad2;
            if (pass == 1) {
#pragma unroll
                for (int i = 0; i < NL; i++) A[NL + 4 + i] = vlane(in, i) ^ mk[i];
            }
            A[NL + 4 + (pass == 1 ? NL : 0)] = interleave(0x1Full);
            A[16] ^= interleave(0x8000000000000000ull);
            keccak_f1600_short_il(A);
            if (pass == 0) {
#pragma unroll
                for (int i = 0; i < NL; i++) mk[i] = A[i];
            }
        }
#pragma unroll
        for (int i = 0; i < NL; i++) { out[2 * i] = (uint32_t)A[i]; out[2 * i + 1] = (uint32_t)(A[i] >> 32); }
    }

    // PRF = SHAKE256(SK_SEED || ADRS) (hash_shake256.cu:38-47)
    SPX_DEV static void PRF(uint32_t out[W], const Adrs &a, const KeyRegs<N> &k) {
        uint64_t o[NL];
        uint64_t dummy[1] = {0};
        short_hash<0, NL>(o, k.skseed, a, dummy);
#pragma unroll
        for (int i = 0; i < NL; i++) { out[2 * i] = (uint32_t)o[i]; out[2 * i + 1] = (uint32_t)(o[i] >> 32); }
    }

    // Root of a FORS subtree (see Sha2::fors_subtree)
    template <class S, class T>
    SPX_DEV static void fors_subtree(uint32_t v[W], Adrs &ad, const KeyRegs<N> &k, uint32_t j0, int sub, uint32_t off,
                                     uint32_t *stk, S sec, T node) {
        int sp = 0;
        for (uint32_t jj = 0; jj < 1u << sub; jj++) {
            const uint32_t j = j0 + jj;
            adrs_height(ad, 0);
            adrs_index(ad, off + j);
            uint32_t x[W];
            PRF(x, ad, k);
            sec(j, x);
            F(v, x, ad, k);
            node(0, j, v);
            int hgt = 0;
            while ((jj >> hgt) & 1u) {   // merge equal-height nodes on the stack
                sp--;
#pragma unroll
                for (int q = 0; q < W; q++) x[q] = stk[sp * W + q];
                hgt++;
                adrs_height(ad, hgt);
                adrs_index(ad, (j >> hgt) + (off >> hgt));
                H(v, x, v, ad, k);
                node(hgt, j >> hgt, v);
            }
#pragma unroll
            for (int q = 0; q < W; q++) stk[sp * W + q] = v[q];
            sp++;
        }
    }

    // T_l streaming: PUB_SEED || ADRS || v_0 || v_1 ...  (lanes, rate 17)
    // buf: per-thread shared memory, kSmemWords words (17 lanes + robust mask block)
    static constexpr int kSmemWords = 2 * 17 + (ROBUST ? 2 * 17 : 0);
    struct TStream {
        uint64_t A[25];
        uint64_t *buf;   // 17 lanes
        int pos;         // lanes filled in buf
        // robust: mask sponge squeezed 17 lanes at a time
        uint64_t M[25];
        int mpos;
    };
    SPX_DEV static void t_init(TStream &t, uint32_t *smem, const KeyRegs<N> &k, const Adrs &a) {
        t.buf = reinterpret_cast<uint64_t *>(smem);
#pragma unroll
        for (int i = 0; i < 25; i++) t.A[i] = 0;
        uint64_t al[4];
        adrs_lanes(a, al);
#pragma unroll
        for (int i = 0; i < NL; i++) t.buf[i] = vlane(k.pub, i);
#pragma unroll
        for (int i = 0; i < 4; i++) t.buf[NL + i] = al[i];
        t.pos = NL + 4;
        if (ROBUST) {
            // mask = SHAKE256(PUB_SEED || ADRS, .): absorb + first permutation
#pragma unroll
            for (int i = 0; i < 25; i++) t.M[i] = 0;
#pragma unroll
            for (int i = 0; i < NL; i++) t.M[i] = vlane(k.pub, i);
#pragma unroll
            for (int i = 0; i < 4; i++) t.M[NL + i] = al[i];
            t.M[NL + 4] = 0x1Full;
            t.M[16] ^= 0x8000000000000000ull;
            keccak_f1600(t.M);
            uint64_t *mb = t.buf + 17;
#pragma unroll
            for (int i = 0; i < 17; i++) mb[i] = t.M[i];
            t.mpos = 0;
        }
    }
    SPX_DEV static void t_flush(TStream &t) {
#pragma unroll
        for (int i = 0; i < 17; i++) t.A[i] ^= t.buf[i];
        keccak_f1600(t.A);
    }
    SPX_DEV static void t_lane(TStream &t, uint64_t x) {
        if (ROBUST) {
            uint64_t *mb = t.buf + 17;
            if (t.mpos == 17) {
                keccak_f1600(t.M);
#pragma unroll
                for (int i = 0; i < 17; i++) mb[i] = t.M[i];
                t.mpos = 0;
            }
            x ^= mb[t.mpos++];
        }
        t.buf[t.pos++] = x;
        if (t.pos == 17) {
            t_flush(t);
            t.pos = 0;
        }
    }
    SPX_DEV static void t_absorb(TStream &t, const uint32_t v[W], const KeyRegs<N> &) {
#pragma unroll
        for (int i = 0; i < NL; i++) t_lane(t, vlane(v, i));
    }
    SPX_DEV static void t_final(uint32_t out[W], TStream &t) {
        for (int i = t.pos; i < 17; i++) t.buf[i] = 0;
        t.buf[t.pos] ^= 0x1Full;
        t.buf[16] ^= 0x8000000000000000ull;
        t_flush(t);
#pragma unroll
        for (int i = 0; i < NL; i++) { out[2 * i] = (uint32_t)t.A[i]; out[2 * i + 1] = (uint32_t)(t.A[i] >> 32); }
    }

    // T_l of M n-byte values: PUB_SEED || ADRS || values, block by block.
    // ld(q) gives lane q of the values.  A robust set's mask lane q belongs to
    // value lane q, so block j takes mask blocks j - 1 and j.
    template <int M, class LD>
    SPX_DEV static void t_values(uint32_t out[W], const KeyRegs<N> &k, const Adrs &a, LD ld) {
        constexpr int PL = NL + 4, Q = M * NL, NB = (PL + Q) / 17 + 1, MB = (Q + 16) / 17;
        uint64_t A[25], S[25], last[PL];   // last: the mask block before's last PL lanes
        uint64_t al[4];
        adrs_lanes(a, al);
#pragma unroll
        for (int i = 0; i < 25; i++) A[i] = S[i] = 0;
        if constexpr (ROBUST) {
#pragma unroll
            for (int i = 0; i < NL; i++) S[i] = vlane(k.pub, i);
#pragma unroll
            for (int i = 0; i < 4; i++) S[NL + i] = al[i];
            S[PL] = 0x1Full;
            S[16] ^= 0x8000000000000000ull;
#pragma unroll
            for (int i = 0; i < PL; i++) last[i] = 0;
        }
#pragma unroll 1
        for (int j = 0; j < NB; j++) {
            if (ROBUST && j < MB) keccak_f1600(S);
#pragma unroll
            for (int i = 0; i < 17; i++) {
                const int q = 17 * j + i - PL;
                uint64_t x = 0;
                if (q >= 0 && q < Q) {
                    const uint2 y = ld((uint32_t)q);
                    x = lane_of(y.x, y.y);
                    if constexpr (ROBUST) x ^= i < PL ? last[i < PL ? i : 0] : S[i - PL < 0 ? 0 : i - PL];
                }
                A[i] ^= x;
            }
            if (ROBUST) {
#pragma unroll
                for (int i = 0; i < PL; i++) last[i] = S[17 - PL + i];
            }
            if (j == 0) {
#pragma unroll
                for (int i = 0; i < NL; i++) A[i] ^= vlane(k.pub, i);
#pragma unroll
                for (int i = 0; i < 4; i++) A[NL + i] ^= al[i];
            }
            if (j == NB - 1) {
                A[(PL + Q) % 17] ^= 0x1Full;
                A[16] ^= 0x8000000000000000ull;
            }
            keccak_f1600(A);
        }
#pragma unroll
        for (int i = 0; i < NL; i++) { out[2 * i] = (uint32_t)A[i]; out[2 * i + 1] = (uint32_t)(A[i] >> 32); }
    }

    // ---- message hashing --------------------------------------------------
    // lane q (little-endian) of m with the SHAKE padding byte 0x1F at mlen;
    // m must be 8-byte aligned and readable up to the next multiple of 8.
    SPX_DEV static uint64_t msg_lane(const uint8_t *m, uint64_t mlen, uint64_t q) {
        uint64_t b = 8 * q;
        if (b + 8 <= mlen) return *reinterpret_cast<const uint64_t *>(m + b);
        if (b > mlen) return 0;
        uint32_t keep = (uint32_t)(mlen - b);  // 0..7
        uint64_t x = keep ? *reinterpret_cast<const uint64_t *>(m + b) : 0ull;
        uint64_t lo = keep ? (0xffffffffffffffffull >> (64 - 8 * keep)) : 0ull;
        return (x & lo) | (0x1Full << (8 * keep));
    }
    // SHAKE256(prefix(P lanes) || m) absorbed into A (state after the last
    // permutation).  Blocks wholly inside the message are loaded one block
    // ahead of the permutation (m + 8 * lane is 8-byte aligned).
    template <int P>
    SPX_DEV static void stream_msg(uint64_t A[25], const uint64_t pre[P], const uint8_t *m, uint64_t mlen) {
        const uint64_t dbytes = 8 * (uint64_t)P + mlen;
        const uint64_t nblocks = dbytes / 136 + 1;
        constexpr int PB = (P + 16) / 17;
        auto full = [&](uint64_t b) { return b >= (uint64_t)PB && 8 * (17 * b - P + 17) <= mlen; };
        uint64_t nxt[17];
        bool have = false;
#pragma unroll
        for (int i = 0; i < 25; i++) A[i] = 0;
        for (uint64_t b = 0; b < nblocks; b++) {
            if (have) {
#pragma unroll
                for (int j = 0; j < 17; j++) A[j] ^= nxt[j];
            } else if (b < PB) {
#pragma unroll
                for (int pb = 0; pb < PB; pb++) {
                    if (pb == (int)b) {
#pragma unroll
                        for (int j = 0; j < 17; j++) {
                            const int g = 17 * pb + j;
                            A[j] ^= g < P ? pre[g < P ? g : 0] : msg_lane(m, mlen, (uint64_t)(g - P));
                        }
                    }
                }
            } else {
                const uint64_t q0 = 17 * b - P;
#pragma unroll
                for (int j = 0; j < 17; j++) A[j] ^= msg_lane(m, mlen, q0 + j);
            }
            have = b + 1 < nblocks && full(b + 1);
            if (have) {
                const uint64_t *p = reinterpret_cast<const uint64_t *>(m + 8 * (17 * (b + 1) - P));
#pragma unroll
                for (int j = 0; j < 17; j++) nxt[j] = p[j];
            }
            // the 0x1F byte comes from msg_lane (the lane holding byte mlen is
            // always inside the last block); the final 0x80 is added here
            if (b == nblocks - 1) A[16] ^= 0x8000000000000000ull;
            keccak_f1600(A);
        }
    }

    // PRF_msg = SHAKE256(SK_PRF || optrand || m, n) (hash_shake256.cu:64-77)
    SPX_DEV static void prf_msg(uint32_t R[W], const uint32_t skprf[W], const uint32_t optrand[W],
                                const uint8_t *m, uint64_t mlen) {
        uint64_t pre[2 * NL], A[25];
#pragma unroll
        for (int i = 0; i < NL; i++) { pre[i] = vlane(skprf, i); pre[NL + i] = vlane(optrand, i); }
        stream_msg<2 * NL>(A, pre, m, mlen);
#pragma unroll
        for (int i = 0; i < NL; i++) { R[2 * i] = (uint32_t)A[i]; R[2 * i + 1] = (uint32_t)(A[i] >> 32); }
    }
    // H_msg = SHAKE256(R || PK || m, dgst) (hash_shake256.cu:96-130)
    SPX_DEV static void h_msg(uint8_t *dg, int dgst_bytes, const uint32_t R[W], const uint32_t pk[2 * W],
                              const uint8_t *m, uint64_t mlen) {
        uint64_t pre[3 * NL], A[25];
#pragma unroll
        for (int i = 0; i < NL; i++) pre[i] = vlane(R, i);
#pragma unroll
        for (int i = 0; i < 2 * NL; i++) pre[NL + i] = vlane(pk, i);
        stream_msg<3 * NL>(A, pre, m, mlen);
        for (int i = 0; i < dgst_bytes; i++) dg[i] = (uint8_t)(A[i >> 3] >> (8 * (i & 7)));
    }
};

}  // namespace cuspx
