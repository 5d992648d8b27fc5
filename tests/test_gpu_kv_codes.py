"""Attention over quantised caches with the codes as matrix operands: queries at the ends of their range (a power of two per head brings them into
fp16), scales that lie on odd addresses, which the kernel with global partials takes, and blocks of a cluster that are done before others."""
import math

import numpy as np
import pytest

from fusekit_b200 import _native as N
from oracle import oracle as O
from tests.helpers import assert_close_bf16, bf
from tests.test_gpu_kernels import normal

pytestmark = pytest.mark.gpu
T = N.Task.make


def case(rt, bits, nq, nkv, hd, cap, pos, up, odd, again=0):
    """Queries times 2^up with keys' scales and biases times 2^-up: the scores stay as they are."""
    rows, per, ng = nkv * cap, 32 // bits, hd // 64
    rng = np.random.default_rng(hd + bits + pos)
    kp, vp = (rng.integers(0, 2 ** 32, (rows, hd // per), dtype=np.uint64).astype(np.uint32) for _ in range(2))
    top = 2 ** bits - 1
    step = lambda f: O.f32_to_bf16((rng.uniform(2.0, 4.0, (rows, ng)) / top * rng.choice([-1.0, 1.0], (rows, ng)) * f).astype(np.float32))
    ks, vs = step(2.0 ** -up), step(1.0)
    kb, vb = (O.f32_to_bf16((-0.4 * top * bf(s)).astype(np.float32)) for s in (ks, vs))
    q = O.f32_to_bf16((bf(normal(f"kc{nq}", nq * hd)) * np.float32(2.0) ** up).astype(np.float32))
    put = lambda a: rt.to_device(np.concatenate([np.zeros(1, np.uint16), a.reshape(-1)])) + 2 if odd else rt.to_device(a)
    bufs = {0: rt.to_device(q), 1: rt.to_device(kp), 2: rt.to_device(vp), 3: rt.alloc(nq * hd * 2), 4: rt.alloc(nq * (cap // 32 + 1) * (hd + 2) * 4), 5: rt.alloc(nkv * 4),
            6: put(ks), 7: put(kb), 8: put(vs), 9: put(vb)}
    rt.state_set(0, pos)
    rt.launch(T(N.TASK_SDPA_DECODE_QUANT, 0, bufs, [nq, nkv, hd, cap, bits], [1.0 / math.sqrt(hd)]))
    first = rt.download(bufs[3], (nq * hd,), np.uint16)
    for _ in range(again):
        rt.launch(T(N.TASK_SDPA_DECODE_QUANT, 0, bufs, [nq, nkv, hd, cap, bits], [1.0 / math.sqrt(hd)]))
        assert np.array_equal(rt.download(bufs[3], (nq * hd,), np.uint16), first)
    want = O.sdpa_decode_quant(q, kp, ks, kb, vp, vs, vb, nq, nkv, hd, cap, min(pos + 1, cap), 1.0 / math.sqrt(hd), bits)
    assert_close_bf16(first, want, f"q{bits}")
    for i, p in bufs.items():
        N.check(rt.L.fk_free(rt.h, p - 2 if odd and i >= 6 else p), "fk_free")


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (28, 4, 128), (4, 2, 256)])
@pytest.mark.parametrize("up", [-60, 0, 60])
def test_queries_of_any_size(runtime, bits, nq, nkv, hd, up):
    for pos in (0, 15, 16, 129, 412):
        case(runtime, bits, nq, nkv, hd, 413, pos, up, False)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("nq,nkv,hd", [(14, 2, 64), (28, 4, 128), (4, 2, 256)])
def test_scales_on_odd_addresses(runtime, bits, nq, nkv, hd):
    """Rows of one group (64 dimensions) are read by themselves and may lie anywhere; those of two and four go to the kernel with global partials."""
    case(runtime, bits, nq, nkv, hd, 201, 150, 0, True)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("nq,nkv,hd,cap", [(1, 1, 64, 2048), (14, 2, 64, 2048), (28, 4, 128, 2048), (4, 2, 256, 2048), (56, 8, 128, 512)])
def test_blocks_of_a_cluster_that_finish_first(runtime, bits, nq, nkv, hd, cap):
    """Blocks without a key, or with fewer rounds of them, hand their share over while others of the cluster (16 blocks, or 8) still read their
    queries: every launch gives the same bits, those of the oracle's grade (``case``)."""
    rt = runtime
    for pos in (0, 17, 300, cap - 1):
        case(rt, bits, nq, nkv, hd, cap, pos, 0, False, again=60)
