"""Small batches (one ciphertext per CTA or per cluster of two) against the throughput kernels and the
oracle: the gate words are the same integers; the CBS rotation stays within the grouped form's
phase-error bound of the exact one.  Batches around SMs / 2 and the SM count."""
from __future__ import annotations

import numpy as np
import pytest

from cbs_harness import OracleCbs
from conftest import load_oracle, load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available()
    return load_pkg(), load_oracle(), torch


def sms(torch):
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("N,n,levels,bg", [(1024, 33, 3, 7), (2048, 21, 3, 7), (1024, 10, 2, 8), (2048, 11, 2, 8)])
def test_gate_words_equal_throughput_form(env, N, n, levels, bg):
    pkg, _, torch = env
    p = pkg.gate_default_params()
    p.N, p.n, p.levels, p.bg_bits = N, n, levels, bg
    full = sms(torch) + 1  # one more than the SMs: the throughput kernel
    ctx = pkg.GateContext(p, max_batch=full)
    ctx.keygen(8)
    ctx.set_multibit(2)
    rng = np.random.default_rng(N + n)
    a = rng.integers(0, 2 ** 32, (full, n), dtype=np.uint64).astype(np.uint32)
    a[0, :2] = 0  # a group without rotations
    b = rng.integers(0, 2 ** 32, full, dtype=np.uint64).astype(np.uint32)
    da, db = (torch.from_numpy(v.view(np.int32)).cuda() for v in (a, b))

    def ext_of(count):
        ext = torch.full((count + 1, N + 1), -1, dtype=torch.int32, device="cuda")
        pkg.call("cbs_gate_bootstrap_batch_device", ctx.handle, da.data_ptr(), db.data_ptr(), count, ext.data_ptr(),
                 None, None, None)
        assert int(ext[count].min()) == -1
        return ext[:count].cpu().numpy()

    want = ext_of(full)
    for count in (1, sms(torch) // 2, sms(torch) // 2 + 1, sms(torch)):
        assert np.array_equal(ext_of(count), want[:count])
    ctx.close()


@pytest.mark.parametrize("preset,N,n,bound", [("3x12", 2048, 31, 33), ("2x18", 2048, 30, 39), ("3x12", 1024, 9, 33)])
@pytest.mark.parametrize("count", [1, 75])  # a cluster of two per ciphertext / one CTA
def test_cbs_phase_error(env, preset, N, n, bound, count):
    pkg, o, torch = env
    p = pkg.preset_params(preset)
    p.N, p.n = N, n
    ctx = pkg.Context(p, max_batch=count)
    ctx.keygen(4)
    ctx.set_br_backend(pkg.BR_FFT64)
    ctx.set_br_multibit(2)
    oc = OracleCbs(o, p, ctx.export_keys())
    rng = np.random.default_rng(count)
    a = rng.integers(0, p.q_lwe, (count, n), dtype=np.uint64)
    b = rng.integers(0, p.q_lwe, count, dtype=np.uint64)
    mv = torch.zeros((count, p.num_lut, 2, N), dtype=torch.int64, device="cuda")
    da, db = (torch.from_numpy(v.view(np.int64)).cuda() for v in (a, b))
    pkg.call("cbs_blind_rotate_batch_device", ctx.handle, da.data_ptr(), db.data_ptr(), count, n, mv.data_ptr(), None)
    got = mv.cpu().numpy().view(np.uint64)
    for i in {0, count - 1}:
        want = oc.br_acc_mb(a[i:i + 1], b[i:i + 1], ctx.export_mb_bsk(), 2)[0]
        # MV output 0 is the finalized accumulator (scaled by N^-1): compare phases times N
        d = oc.phase_coef(got[i, 0]) - oc.phase_coef(want)
        err = max(abs((int(x) * N + p.Q // 2) % p.Q - p.Q // 2) for x in d)
        assert err < 2 ** bound
    ctx.close()
