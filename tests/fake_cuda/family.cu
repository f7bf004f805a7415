// Hash families for the host-memory runtime: "signatures" that show which
// inputs they were made from.  A signature is the randomiser (0xad without
// one), then SK_PRF of its key row; a verdict is 0 for a signature of the
// right length (or without one to look at) whose second n bytes are PUB_SEED.
#include "../../cuspx_gb300/csrc/spx_launch.cuh"
#include "fake_cuda.h"

namespace cuspx {
namespace {
const uint8_t *key_row(const KeyRef &k, uint32_t i, int dev) {
    uint32_t r = i;
    if (k.keyrow) r = fake_access(k.keyrow + i, 4, dev) ? k.keyrow[i] : 0;
    const uint8_t *p = k.keys + (uint64_t)r * k.stride;
    return fake_access(p, k.stride, dev) ? p : nullptr;
}
void sign(const SetParams &P, SignArgs A, const Tuning &, cudaStream_t s, PhaseTimer *, uint64_t, const StreamFork *) {
    const int dev = fake_stream_device(s);
    fake_launch([=] {
        for (uint32_t i = 0; i < A.count; i++) {
            uint8_t *sig = A.sig + (uint64_t)i * P.sig_bytes;
            const uint8_t *sk = key_row(A.sk, i, dev);
            if (!sk || !fake_access(sig, P.sig_bytes, dev) || !fake_access(A.status + i, 4, dev) ||
                !fake_access(A.msg.off + i, 8, dev) || !fake_access(A.msg.len + i, 8, dev))
                return;
            memset(sig, 0xad, P.n);
            if (A.optrand && fake_access(A.optrand + i * P.n, P.n, dev)) memcpy(sig, A.optrand + i * P.n, P.n);
            memcpy(sig + P.n, sk + P.n, P.n);
            A.status[i] = 0;
        }
    });
}
void verify(const SetParams &P, const VerifyArgs &B, const Tuning &, cudaStream_t s, PhaseTimer *, uint64_t,
            const VerifyLists *, const VerifyFork *) {
    const int dev = fake_stream_device(s);
    const VerifyArgs A = B;
    fake_launch([=] {
        for (uint32_t i = 0; i < A.count; i++) {
            const uint8_t *sig = A.sig + (uint64_t)i * A.sig_stride, *pk = key_row(A.pk, i, dev);
            if (!pk || !fake_access(sig, P.sig_bytes, dev) || !fake_access(A.verdict + i, 4, dev)) return;
            bool ok = !memcmp(sig + P.n, pk, P.n);
            if (A.siglen) ok &= fake_access(A.siglen + i, 8, dev) && A.siglen[i] == (uint64_t)P.sig_bytes;
            A.verdict[i] = ok ? 0 : -1;
        }
    });
}
void keygen(const SetParams &, const KeygenArgs &, const Tuning &, cudaStream_t, PhaseTimer *) {}
cudaError_t configure() { return cudaSuccess; }
void fill(int h, int n, int r) {
    FamilyOps &o = g_family[h][n / 8 - 2][r];
    o.configure = &configure;
    o.sign = &sign;
    o.verify = &verify;
    o.keygen = &keygen;
    o.smem_words = 1;
}
}  // namespace
#define FAMILY(h, n, r) \
    void register_family_##h##_##n##_##r() { fill(h, n, r); }
FAMILY(0, 16, 0) FAMILY(0, 16, 1) FAMILY(0, 24, 0) FAMILY(0, 24, 1) FAMILY(0, 32, 0) FAMILY(0, 32, 1)
FAMILY(1, 16, 0) FAMILY(1, 16, 1) FAMILY(1, 24, 0) FAMILY(1, 24, 1) FAMILY(1, 32, 0) FAMILY(1, 32, 1)
}  // namespace cuspx
