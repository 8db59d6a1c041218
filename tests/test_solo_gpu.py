"""The mb = 2 blind-rotation forms by batch: one ciphertext per CTA or per cluster of two (small batches
and what a wave leaves over) and two per lane set.  Gate words: equal to the oracle's exact grouped
rotation and the same in every form.  CBS: within the grouped form's phase-error bound of the exact
rotation.  Batches around SMs / 2, the SM count and the wave sizes."""
from __future__ import annotations

import numpy as np
import pytest

from cbs_harness import OracleCbs
from conftest import load_oracle, load_pkg
from gate_harness import OracleGate, declare_gate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available()
    return load_pkg(), load_oracle(), torch


def sms(torch):
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("N,n,levels,bg", [(1024, 33, 3, 7), (2048, 21, 3, 7), (1024, 10, 2, 8), (2048, 11, 2, 8)])
def test_gate_words_in_every_form(env, N, n, levels, bg):
    pkg, o, torch = env
    p = pkg.gate_default_params()
    p.N, p.n, p.levels, p.bg_bits = N, n, levels, bg
    S = sms(torch)
    counts = (1, 2, S // 2, S // 2 + 1, S, S + 1, 2 * S, 2 * S + 1, 4 * S + 3)
    full = counts[-1]
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
        return ext[:count].cpu().numpy().view(np.uint32)

    got = [ext_of(c) for c in counts]
    for g in got[:-1]:
        assert np.array_equal(g, got[-1][:len(g)])
    pick = [0, 1, S, 2 * S, full - 1]
    want = OracleGate(declare_gate(o), p, ctx.export_keys()).blind_rotate_mb(a[pick], b[pick], ctx.export_mb_bsk(), 2)
    assert np.array_equal(got[-1][pick], want)
    # a persistent grid (fewer CTAs than ciphertexts) through the request table: the same outputs
    count = 2 * S + 7
    outs = []
    for grid in (0, 5):
        oa = torch.zeros((count, n), dtype=torch.int32, device="cuda")
        ob = torch.zeros(count, dtype=torch.int32, device="cuda")
        half = count // 2
        ctx.ragged_plan([(da.data_ptr(), db.data_ptr(), oa.data_ptr(), ob.data_ptr(), half),
                         (da[half:].data_ptr(), db[half:].data_ptr(), oa[half:].data_ptr(), ob[half:].data_ptr(),
                          count - half)], grid_ctas=grid)
        ctx.ragged_launch()
        outs.append((oa.cpu().numpy(), ob.cpu().numpy()))
    assert all(np.array_equal(x, y) for x, y in zip(*outs))
    ctx.close()


@pytest.mark.parametrize("preset,N,n,bound", [("3x12", 2048, 31, 33), ("2x18", 2048, 30, 39), ("3x12", 1024, 9, 33)])
def test_cbs_phase_error(env, preset, N, n, bound):
    pkg, o, torch = env
    p = pkg.preset_params(preset)
    p.N, p.n = N, n
    S = sms(torch)
    full = 2 * S + 9
    ctx = pkg.Context(p, max_batch=full)
    ctx.keygen(4)
    ctx.set_br_backend(pkg.BR_FFT64)
    ctx.set_br_multibit(2)
    oc, mbk = OracleCbs(o, p, ctx.export_keys()), ctx.export_mb_bsk()
    rng = np.random.default_rng(n)
    a = rng.integers(0, p.q_lwe, (full, n), dtype=np.uint64)
    b = rng.integers(0, p.q_lwe, full, dtype=np.uint64)
    pick = [0, S // 2, S, full - 1]
    want = {i: oc.phase_coef(oc.br_acc_mb(a[i:i + 1], b[i:i + 1], mbk, 2)[0]) for i in pick}
    da, db = (torch.from_numpy(v.view(np.int64)).cuda() for v in (a, b))
    # clusters of two, one CTA each, two per CTA with an odd last, the split batch
    for count in (1, S // 2 + 1, S + 1, full):
        mv = torch.full((count + 1, p.num_lut, 2, N), -1, dtype=torch.int64, device="cuda")
        pkg.call("cbs_blind_rotate_batch_device", ctx.handle, da.data_ptr(), db.data_ptr(), count, n, mv.data_ptr(),
                 None)
        assert int(mv[count].max()) == -1
        got = mv[:count].cpu().numpy().view(np.uint64)
        for i in (i for i in pick if i < count):
            # MV output 0 is the finalized accumulator (scaled by N^-1): compare phases times N
            d = oc.phase_coef(got[i, 0]) - want[i]
            assert max(abs((int(x) * N + p.Q // 2) % p.Q - p.Q // 2) for x in d) < 2 ** bound
    ctx.close()
