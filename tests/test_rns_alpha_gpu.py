"""Hybrid key switch over the number of special primes (alpha: the base conversions are compiled
for 1, 2, 4, 8 and 16 terms) and over the alignment of the caller's key pointers (the inner product
takes two coefficients per 16-byte word where it can), against the CPU oracle: bit-exact, with
residues of q - 1 among the inputs, where the FP64 sums are largest."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_pkg, load_oracle
from rns_harness import declare_rns, rns_primes

pytestmark = pytest.mark.gpu


def limbs_of(rng, mods, n):
    x = np.stack([rng.integers(0, int(m), n, dtype=np.uint64) for m in mods])
    top = rng.random(x.shape) < 0.5
    return np.where(top, np.asarray(mods, np.uint64)[:, None] - np.uint64(1), x)


@pytest.mark.parametrize("logn,size_q,alpha,shift", [
    (10, 3, 1, 0), (10, 5, 2, 1), (10, 7, 3, 0), (11, 9, 4, 1), (10, 11, 5, 0), (10, 17, 8, 0), (10, 19, 9, 1),
    (10, 17, 16, 0), (13, 18, 16, 1), (13, 3, 2, 0)])
def test_keyswitch_by_alpha_and_alignment(logn, size_q, alpha, shift):
    import torch
    pkg, o = load_pkg(), declare_rns(load_oracle())
    n, count = 1 << logn, 5  # five ciphertexts: a full group of four and a remainder
    q, p = rns_primes(o, n, size_q, alpha)
    chain = np.concatenate([q, p])
    rng = np.random.default_rng(100 * alpha + shift)
    beta = -(-size_q // alpha)
    c2 = np.stack([limbs_of(rng, q, n) for _ in range(count)])
    ct = np.stack([[limbs_of(rng, q, n) for _ in range(2)] for _ in range(count)])
    evk = np.stack([[limbs_of(rng, chain, n) for _ in range(2)] for _ in range(beta)])
    ctx = pkg.RnsContext(n, q, p)

    def dev(a, off=0):
        flat = torch.zeros(a.size + off, dtype=torch.int64)
        flat[off:] = torch.from_numpy(np.ascontiguousarray(a).view(np.int64).reshape(-1))
        return flat.cuda()[off:]

    d_ct, d_c2 = dev(ct), dev(c2)
    d_evk = [dev(e, shift) for e in evk]  # shift = 1: keys that start on an odd 8-byte word
    assert all((t.data_ptr() % 16 != 0) == bool(shift) for t in d_evk)
    ptrs = pkg.RnsContext.evk_array([t.data_ptr() for t in d_evk])
    pkg.call("cbs_rns_keyswitch_inplace", ctx.handle, d_ct.data_ptr(), d_c2.data_ptr(), ptrs, size_q, count, None)
    torch.cuda.synchronize()
    got = d_ct.cpu().numpy().view(np.uint64).reshape(ct.shape)
    for k in range(count):
        want = np.ascontiguousarray(ct[k]).copy()
        o.orc_keyswitch(want, np.ascontiguousarray(c2[k]), np.ascontiguousarray(evk), logn, q, size_q, size_q, p,
                        alpha)
        assert np.array_equal(got[k], want)
    ctx.close()
