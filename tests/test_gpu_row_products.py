"""Products of many rows at the sizes of whole prompts (rings that wrap many times, several tiles a block, ragged last rows and columns) against 64 bits, and
the prompts that they serve: the answer comes, pass after pass the same one, and is that of short portions."""
import numpy as np
import pytest
import torch

from fusekit_b200 import _native as N
from fusekit_b200.layered import LayeredEngine
from fusekit_b200.model_spec import config
from tests import layered_models as LM
from tests.test_gpu_layered import check_logits

pytestmark = pytest.mark.gpu
T = N.Task.make


def rows_of(rt, t):
    return rt.to_device(t.to(torch.bfloat16).contiguous().view(torch.int16).cpu().numpy().view(np.uint16).reshape(-1))


def weight_of(rt, w):
    wid = rt.weight_alloc(*w.shape, 16)
    rt.weight_upload_rows(wid, 0, w.contiguous().view(torch.int16).cpu().numpy().view(np.uint16))
    rt.weight_keep_rows(wid)
    return wid


def case(m, n, k):
    gen = torch.Generator().manual_seed(m + n + k)
    return tuple(torch.randn(shape, generator=gen).to(torch.bfloat16) for shape in ((m, k), (n, k)))


def worst(got, want, k, half):
    """Largest error over its bound: k products of unit size summed in 32 bits, cut at worst (2^-23 of a partial sum, which stays below 6 sqrt(k), at each of
    k / 16 steps), then half a last place of bf16."""
    bound = k / 16 * 2.0 ** -23 * 6 * k ** 0.5 + (2.0 ** -8 * want.abs() if half else 0.0)
    return ((got.double() - want).abs() / bound).max().item()


# 32 and 80 slices of 64 columns, five tiles a block, one row and one column past a tile; many launches behind one another
@pytest.mark.parametrize("m,n,k", [(2048, 3088, 2048), (1500, 2560, 5120), (2048, 12000, 512), (2049, 2561, 2048), (190, 9000, 2048)])
def test_plain_rows_of_whole_prompts(runtime, m, n, k):
    rt = runtime
    x, w = case(m, n, k)
    xd, wid, ldy = rows_of(rt, x), weight_of(rt, w), -(-n // 8) * 8
    y, yf = rt.alloc(m * ldy * 2), rt.alloc(m * n * 4)
    rt.state_set(0, 0)
    half = T(N.TASK_LINEAR_ROWS, -1, {0: xd, 1: wid, 2: y}, [m, 0, n, k, ldy, 0, 0, 0])
    full = T(N.TASK_LINEAR_ROWS, -1, {0: xd, 1: wid, 2: yf}, [m, 0, n, k, n, 0, 256, 0])
    tasks = (N.Task * 40)(*([half, full] * 20))
    N.check(rt.L.fk_launch_batch(rt.h, tasks, 40), "fk_launch_batch")
    assert rt.state_get()[2] == 0
    want = (x.cuda().double() @ w.cuda().double().T).cpu()
    assert worst(torch.from_numpy(rt.download(yf, (m, n), np.float32)), want, k, False) <= 1
    got = torch.from_numpy(rt.download(y, (m, ldy), np.uint16).view(np.int16)).view(torch.bfloat16)[:, :n]
    assert worst(got, want, k, True) <= 1
    for p in (xd, y, yf):
        N.check(rt.L.fk_free(rt.h, p), "fk_free")


# every kind of column: SiLU, plain, 32-bit and (gate, up) pairs
@pytest.mark.parametrize("m,k,silu,plain,exact,pairs", [(1500, 5120, 512, 4096, 4128, 2048), (2049, 2048, 96, 4160, 4192, 3001)])
def test_block_rows_of_whole_prompts(runtime, m, k, silu, plain, exact, pairs):
    rt, n, limit, ld3 = runtime, exact + 2 * pairs, 7.0, -(-pairs // 8) * 8
    x, w = case(m, n, k)
    w = (w.float() * k ** -0.5).to(torch.bfloat16)
    xd, wid = rows_of(rt, x), weight_of(rt, w)
    y, z, ff = rt.alloc(m * plain * 2), rt.alloc(m * (exact - plain) * 4), rt.alloc(m * ld3 * 2)
    rt.state_set(0, 0)
    tasks = (N.Task * 20)(*[T(N.TASK_BLOCK_LINEAR_ROWS, 0, {0: xd, 1: wid, 2: y, 3: z, 4: ff}, [m, plain, exact, n, plain, ld3, 0, silu], [limit])] * 20)
    N.check(rt.L.fk_launch_batch(rt.h, tasks, 20), "fk_launch_batch")
    assert rt.state_get()[2] == 0
    want = (x.cuda().double() @ w.cuda().double().T).cpu()
    bf = lambda p, ld, c: torch.from_numpy(rt.download(p, (m, ld), np.uint16).view(np.int16)).view(torch.bfloat16)[:, :c]      # noqa: E731
    step = 2.0 ** -23 * k / 16 * 6                      # sums of unit size
    assert ((torch.from_numpy(rt.download(z, (m, exact - plain), np.float32)).double() - want[:, plain:exact]).abs() <= step).all()
    got = bf(y, plain, plain).double()
    some = want[:, :plain].clone()
    some[:, :silu] = torch.nn.functional.silu(some[:, :silu])
    assert ((got - some).abs() <= 2.0 ** -8 * some.abs() + 1.1 * step).all()       # the slope of SiLU is at most 1.1
    from oracle import layered as OL
    glu = torch.from_numpy(OL.clamped_glu(want[:, exact::2].numpy(), want[:, exact + 1::2].numpy(), limit))
    assert ((bf(ff, ld3, pairs).double() - glu).abs() <= 2.0 ** -8 * glu.abs() + 16 * step).all()      # both factors' errors times the other, below 8 each
    for p in (xd, y, z, ff):
        N.check(rt.L.fk_free(rt.h, p), "fk_free")


@pytest.mark.parametrize("name,tokens,forced", [("fatulix-2048", 2048, 0), ("kakunex-2048", 190, 3), ("kakunex-5120", 1500, 0)])
def test_whole_prompts_answer_every_time(name, tokens, forced):
    spec = config(name)
    eng = LayeredEngine(spec, tokens + forced)
    try:
        eng.load_synthetic()
        if forced:
            eng.capture()
        ids = np.random.default_rng(tokens).integers(0, spec.vocab, tokens + forced).astype(np.uint32)
        want = list(range(tokens // 40, tokens, tokens // 20))
        seen = None
        for _ in range(30):
            got = [eng.step(ids[:tokens], 0, want)] + [eng.step(ids[t:t + 1], t, [0]) for t in range(tokens, tokens + forced)]
            assert all(np.isfinite(a).all() for a in got)
            assert seen is None or all(np.array_equal(a, b) for a, b in zip(got, seen))
            seen = got
        eng.max_rows = 60                               # portions of few rows take other kernels
        check_logits(seen[0], eng.step(ids[:tokens], 0, want), "bfloat16", name)
    finally:
        eng.close()
