"""The tensor-core key switches (one-hot x byte-plane products) against the oracle's key switches,
word for word, at the edges of their tiles: items around multiples of 16 and 128, output words
around multiples of 128, every digit width with a kernel, slot counts that do not fill a step."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from cbs_harness import OracleCbs
from conftest import load_oracle, load_pkg
from gate_harness import OracleGate, declare_gate
from tcb_harness import OracleTcb, declare_tcb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    assert torch.cuda.is_available()
    return load_pkg(), load_oracle(), torch


def fault(pkg):
    v = ctypes.c_uint32()
    pkg.call("cbs_keyswitch_device_fault", ctypes.byref(v), 0)
    return v.value


@pytest.mark.parametrize("n,bits,levels,counts", [
    (3, 2, 8, (1, 15, 16, 17)), (126, 2, 8, (127, 128)), (127, 1, 5, (129,)), (128, 3, 7, (33,)),
    (4, 4, 3, (257,)), (636, 2, 8, (2,)), (5, 5, 3, (4,)), (6, 7, 2, (20,)), (5, 8, 2, (4,))])  # 8: the gather kernel
def test_gate_keyswitch_words(env, n, bits, levels, counts):
    pkg, o, torch = env
    p = pkg.gate_default_params()
    p.n, p.ks_base_bits, p.ks_levels = n, bits, levels
    ctx = pkg.GateContext(p, max_batch=300)
    ctx.keygen(50 + n)
    og = OracleGate(declare_gate(o), p, ctx.export_keys())
    rng = np.random.default_rng(n)
    for count in counts:
        a = torch.from_numpy(rng.integers(0, 2 ** 32, (count, n), dtype=np.uint64).astype(np.uint32).view(np.int32)).cuda()
        b = torch.from_numpy(rng.integers(0, 2 ** 32, count, dtype=np.uint64).astype(np.uint32).view(np.int32)).cuda()
        ext = torch.zeros((count, p.N + 1), dtype=torch.int32, device="cuda")
        oa = torch.full((count + 1, n), -1, dtype=torch.int32, device="cuda")
        ob = torch.full((count + 1,), -1, dtype=torch.int32, device="cuda")
        pkg.call("cbs_gate_bootstrap_batch_device", ctx.handle, a.data_ptr(), b.data_ptr(), count, ext.data_ptr(),
                 oa.data_ptr(), ob.data_ptr(), None)
        wa, wb = og.keyswitch(ext.cpu().numpy().view(np.uint32))
        assert np.array_equal(oa[:count].cpu().numpy().view(np.uint32), wa)
        assert np.array_equal(ob[:count].cpu().numpy().view(np.uint32), wb)
        assert int(oa[count].min()) == -1 and int(ob[count]) == -1  # nothing past the batch
    assert fault(pkg) == 0
    ctx.close()


@pytest.mark.parametrize("n,qks_bits,base_bits,counts", [
    (20, 14, 7, (1, 16, 130)), (127, 10, 5, (3,)), (128, 12, 6, (17,)), (630, 16, 8, (5,)), (9, 8, 4, (6,)), (130, 14, 7, (257,))])
def test_extract_keyswitch_words(env, n, qks_bits, base_bits, counts):
    pkg, o, torch = env
    p = pkg.default_params()
    p.N, p.n, p.qks, p.base_ks = 1024, n, 1 << qks_bits, 1 << base_bits
    ctx = pkg.Context(p, max_batch=4)
    ctx.keygen(9)
    oc = OracleCbs(o, p, ctx.export_keys())
    rng = np.random.default_rng(qks_bits)
    words = rng.integers(0, p.Q, (3, 2, p.N), dtype=np.uint64)
    words[0, 0, :8] = 0
    dw = torch.from_numpy(words.view(np.int64)).cuda()
    for count in counts:
        idx = rng.integers(0, p.N, count)
        idx[0], idx[-1] = 0, p.N - 1
        info = ((rng.integers(0, 3, count) << 16) | idx).astype(np.uint32)
        oa = torch.full((count, n + 3), -1, dtype=torch.int64, device="cuda")
        ob = torch.full((count,), -1, dtype=torch.int64, device="cuda")
        pkg.call("cbs_extract_keyswitch_device", ctx.handle, dw.data_ptr(), 3, info.ctypes.data, count, oa.data_ptr(),
                 ob.data_ptr(), n + 3, None)
        wa, wb = oc.extract(words, info)
        assert np.array_equal(oa[:, :n].cpu().numpy().view(np.uint64), wa)
        assert np.array_equal(ob.cpu().numpy().view(np.uint64), wb)
        assert int(oa[:, n:].max()) == -1  # the stride's gap is untouched
    assert fault(pkg) == 0
    ctx.close()


@pytest.mark.parametrize("base_bits,counts", [(2, (1, 6)), (4, (43,)), (8, (2,))])  # 8: the gather kernel
def test_pfks_words(env, base_bits, counts):
    pkg, o, torch = env
    p = pkg.tcb_default_params()
    p.n, p.N2, p.N1, p.pfks_base_bits, p.pfks_levels = 6, 1024, 256, base_bits, 32 // base_bits
    ctx = pkg.TcbContext(p, max_batch=64)
    ctx.keygen(21)
    ot = OracleTcb(declare_tcb(o), p, ctx.export_keys(with_pfks=True))
    for count in counts:
        a, b = ctx.encrypt(np.arange(count) % 2, seed=3)
        da, db = (torch.from_numpy(v.view(np.int32)).cuda() for v in (a, b))
        ext = torch.zeros((count, p.cb_levels, p.N2 + 1), dtype=torch.int64, device="cuda")
        rgsw = torch.full((count + 1, p.cb_levels, 2, 2, p.N1), -1, dtype=torch.int32, device="cuda")
        pkg.call("cbs_tcb_circuit_bootstrap_device", ctx.handle, da.data_ptr(), db.data_ptr(), count, ext.data_ptr(),
                 rgsw.data_ptr(), None)
        want = ot.pfks(ext.cpu().numpy().view(np.uint64))
        assert np.array_equal(rgsw[:count].cpu().numpy().view(np.uint32), want)
        assert int(rgsw[count].min()) == -1 and int(rgsw[count].max()) == -1
    assert fault(pkg) == 0
    ctx.close()
