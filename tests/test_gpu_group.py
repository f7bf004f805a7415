"""Mixed-set runs whose batches are replaced by larger ones and used at the old
sizes again, with and without randomisers: byte-identical to the oracle."""
import random

import pytest

pytestmark = pytest.mark.gpu

SETS = ("sha256-128f-simple", "shake256-128f-simple")


def test_mixed_signer_sizes_and_randomisers(engine):
    import cuspx_gb300 as c
    import spx_oracle
    rng = random.Random(21)
    oracles = [spx_oracle.Oracle(s) for s in SETS]
    keys = [o.seed_keypair(rng.randbytes(o.p.seed_bytes)) for o in oracles]
    ms = c.MixedSigner(engine)
    for count, opt in ((2, False), (4, False), (2, False), (2, True), (2, False), (4, True), (4, False), (2, True)):
        which = [i % 2 for i in range(2 * count)]
        msgs = [rng.randbytes(40 + i) for i in range(2 * count)]
        rand = [rng.randbytes(oracles[w].p.n) for w in which] if opt else None
        sigs, status, _ = ms.sign([engine.set_id(SETS[w]) for w in which], [keys[w][1] for w in which], msgs, rand)
        assert not any(status)
        for i, w in enumerate(which):
            assert sigs[i] == oracles[w].sign(msgs[i], keys[w][1], rand[i] if opt else None)
    ms.close()
