"""The typed forms of the frequent training ops (ready-queue kernel) against the general bodies (static kernel): the same bits on the same
input, at the sizes where a typed form changes its instance, its buffering or hands over to the general body."""
import numpy as np
import pytest

from kvm_b200.executor import CFG_DYNAMIC, CFG_STATIC, Executor
from kvm_b200.workloads.graph import Graph

pytestmark = pytest.mark.gpu


def same_bits(g):
    b = g.to_bundle()
    got = []
    for flags in (CFG_DYNAMIC, CFG_STATIC):
        with Executor(flags=flags) as ex:
            ex.load(b)
            assert ex.run().done == len(b.tasks)
            assert ex.plan_info()[0] == (flags == CFG_STATIC)
            got.append({s['name']: ex.read_buffer(s['name']) for s in b.buffers})
    for name, x in got[0].items():
        assert np.array_equal(x.view(np.uint32), got[1][name].view(np.uint32)), name
    return got[0]


def normal(seed, *shape):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


# eight elements are the smallest typed range, 8192 a stage of the stream, four of them its depth; multiples of four only go to the general body
@pytest.mark.parametrize('n', [8, 12, 24, 4096, 8192, 8200, 32768, 40968])
def test_gradnorm_partial(kvm_lib, n):
    g = Graph('gradnorm')
    for i in range(6):
        g.data(f'g{i}', normal(i, 1, n + 8))
        g.buffer(f'p{i}', 1, 2)
        for slot in (0, 1):
            g.task('gradnorm_partial', {'g': f'g{i}', 'partial': f'p{i}', 'slot': slot, 'e0': 8 * slot, 'e1': n + 8 * slot}, [f'g{i}'], [(f'p{i}', (0, 1), (slot, slot + 1))])
    same_bits(g)


# rows around a row group, a stage (64 rows, 128 of a bf16 column sum) and the stages in flight; columns around a block of 64, and too few
# for a 16-byte piece of bf16
@pytest.mark.parametrize('R', [1, 7, 9, 63, 65, 128, 129, 513, 1030])
@pytest.mark.parametrize('D,c0', [(4, 0), (68, 0), (136, 8)])
def test_column_reductions(kvm_lib, R, D, c0):
    g = Graph('columns')
    g.data('x', normal(1, R, D)), g.data('xb', normal(2, R, D), 'bf16'), g.data('dy', normal(3, R, D)), g.data('dyb', normal(4, R, D), 'bf16')
    g.data('mean', normal(5, R, 1)), g.data('rstd', np.abs(normal(6, R, 1)) + 0.5)
    for src in ('x', 'xb'):
        for acc in (0, 1):
            out = g.data(f'sum.{src}.{acc}', normal(7, 1, D))
            g.task('colsum', {'x': src, 'out': out, 'R': R, 'c0': c0, 'c1': D, 'acc': acc}, [src], [out])
    for src, dy in (('x', 'dy'), ('x', 'dyb'), ('xb', 'dy'), ('xb', 'dyb')):
        for acc in (0, 1):
            dg, db = g.data(f'dg.{src}.{dy}.{acc}', normal(8, 1, D)), g.data(f'db.{src}.{dy}.{acc}', normal(9, 1, D))
            g.task('norm_bwd_params', {'x': src, 'dy': dy, 'mean': 'mean', 'rstd': 'rstd', 'dgamma': dg, 'dbeta': db, 'R': R, 'd': D, 'c0': c0, 'c1': D, 'acc': acc}, [src, dy], [dg, db])
    same_bits(g)


# a stage is 2048 float32 or 4096 bf16 elements, four of them in flight; ranges that end inside a stage or start off its grid, outputs in
# place, and ranges that are no multiple of the typed forms' pieces
@pytest.mark.parametrize('e0,e1', [(0, 8), (8, 4104), (0, 4096), (16, 16408), (0, 40960), (4, 5000), (3, 4099)])
def test_elementwise(kvm_lib, e0, e1):
    n = -(-e1 // 8) * 8
    g = Graph('elementwise')
    for dt in ('f32', 'bf16'):
        for place in ('new', 'first', 'second'):
            a, b = g.data(f'a.{dt}.{place}', normal(1, 1, n), dt), g.data(f'b.{dt}.{place}', normal(2, 1, n), dt)
            for op, args in (('residual_add', {'a': a, 'b': b}), ('gelu_bwd', {'x': a, 'dy': b})):
                src = {k: g.data(f'{v}.{op}', normal(3 + i, 1, n), dt) for i, (k, v) in enumerate(args.items())}
                out = g.buffer(f'out.{dt}.{place}.{op}', 1, n, dt) if place == 'new' else list(src.values())[place == 'second']
                extra = {'out': out} if op == 'residual_add' else {'dx': out, 'acc': 0}
                g.task(op, {**src, **extra, 'e0': e0, 'e1': e1}, list(src.values()), [out])
    x, o = g.data('x', normal(5, 1, n)), g.buffer('rounded', 1, n, 'bf16')
    g.task('round_bf16', {'x': x, 'out': o, 'e0': e0, 'e1': e1}, [x], [o])
    same_bits(g)


# widths around the instances (256, 768, 1024 columns) and past them; rows that leave warps without one
@pytest.mark.parametrize('d', [8, 248, 256, 260, 264, 768, 776, 1024, 1032])
@pytest.mark.parametrize('rows', [1, 37])
def test_layernorm(kvm_lib, d, rows):
    g = Graph('layernorm')
    g.data('x', normal(1, rows, d)), g.data('gamma', normal(2, 1, d)), g.data('beta', normal(3, 1, d))
    for dt in ('f32', 'bf16'):
        for n, r, c, t in (('out', rows, d, dt), ('mean', rows, 1, 'f32'), ('rstd', rows, 1, 'f32')):
            g.buffer(f'{n}.{dt}', r, c, t)
        g.task('layernorm_fwd', {'x': 'x', 'gamma': 'gamma', 'beta': 'beta', 'out': f'out.{dt}', 'mean': f'mean.{dt}', 'rstd': f'rstd.{dt}', 'r0': 0, 'r1': rows, 'd': d, 'eps': 1e-5},
               ['x'], [f'out.{dt}', f'mean.{dt}', f'rstd.{dt}'])
        g.data(f'dy.{dt}', normal(4, rows, d), dt)
        for acc in (0, 1):
            dx = g.data(f'dx.{dt}.{acc}', normal(5, rows, d))
            g.task('layernorm_bwd_dx', {'x': 'x', 'dy': f'dy.{dt}', 'gamma': 'gamma', 'mean': f'mean.{dt}', 'rstd': f'rstd.{dt}', 'dx': dx, 'r0': 0, 'r1': rows, 'd': d, 'acc': acc},
                   ['x', f'dy.{dt}', f'mean.{dt}', f'rstd.{dt}'], [dx])
    same_bits(g)


# the shortest typed row, two row buffers, one (more than half of the scratch), and a row too long for one
@pytest.mark.parametrize('V', [1032, 8200, 50304, 65536, 120000])
def test_cross_entropy(kvm_lib, V):
    rows, rng = 5, np.random.default_rng(V)
    g = Graph('ce')
    g.data('logits', normal(1, rows, V), 'bf16'), g.data('tgt', rng.integers(0, V, (rows, 1), dtype=np.int32), 'i32')
    g.buffer('rowloss', rows, 1), g.buffer('lse', rows, 1), g.buffer('dlogits', rows, V, 'bf16')
    for r0, r1 in ((0, 2), (2, 5)):
        g.task('softmax_ce_fused', {'logits': 'logits', 'tgt': 'tgt', 'rowloss': 'rowloss', 'lse': 'lse', 'dlogits': 'dlogits', 'r0': r0, 'r1': r1, 'V': V, 'ignore': -1, 'N': rows, 'scale': 1.0},
               ['logits'], [(n, (r0, r1)) for n in ('rowloss', 'lse', 'dlogits')])
    same_bits(g)


@pytest.mark.parametrize('H,hd', [(1, 32), (3, 64), (5, 128), (12, 64)])
def test_attention_delta(kvm_lib, H, hd):
    T, B = 45, 3
    g = Graph('delta')
    for dt in ('f32', 'bf16'):
        g.data(f'o.{dt}', normal(1, B * T, H * hd), dt), g.data(f'do.{dt}', normal(2, B * T, H * hd), dt), g.buffer(f'delta.{dt}', B * H * T, 1)
        for r0, r1 in ((0, 17), (17, 90), (90, B * T)):
            g.task('attn_bwd_delta', {'o': f'o.{dt}', 'do': f'do.{dt}', 'delta': f'delta.{dt}', 'r0': r0, 'r1': r1, 'T': T, 'H': H, 'hd': hd}, [f'o.{dt}'], [])
    same_bits(g)


@pytest.mark.parametrize('e0,e1', [(0, 4), (4, 2052), (0, 8192), (8, 20004), (2, 4099)])
def test_adamw(kvm_lib, e0, e1):
    n = -(-e1 // 8) * 8
    g = Graph('adamw')
    for i, name in enumerate('pgm'):
        g.data(name, normal(i, 1, n))
    g.data('v', np.abs(normal(9, 1, n))), g.data('clip', np.array([[0.7]], np.float32)), g.data('step', np.array([[3]], np.int32), 'i32')
    g.task('adamw', {'p': 'p', 'g': 'g', 'm': 'm', 'v': 'v', 'gscale': 'clip', 'step': 'step', 'e0': e0, 'e1': e1, 'lr': 1e-3, 'b1': 0.9, 'b2': 0.999, 'eps': 1e-8, 'wd': 0.1},
           ['g', 'clip', 'step'], ['p', 'm', 'v'])
    same_bits(g)


# twenty splits at once in the static kernel's form, more in the op's own; two forms of one sum: float32 roundings of up to 21 terms apart
@pytest.mark.parametrize('S', [1, 20, 21, 30])
def test_merge_of_splits(kvm_lib, S):
    H, hd, rng = 3, 64, np.random.default_rng(S)
    part = rng.standard_normal((S * H, hd + 2)).astype(np.float32)
    part[:, hd + 1] = np.abs(part[:, hd + 1]) + 0.1
    if S > 2:
        part[H:2 * H, hd:] = [-3.4028234663852886e38, 0.0]      # an empty split
    g = Graph('merge')
    g.data('part', part), g.buffer('o', 1, H * hd)
    g.task('attn_decode_merge', {'part': 'part', 'o': 'o', 'b': 0, 'h0': 0, 'h1': H, 'S': S, 'H': H, 'hd': hd}, ['part'], ['o'])
    b = g.to_bundle()
    p = part.reshape(S, H, hd + 2).astype(np.float64)
    e = np.where(p[..., hd + 1] > 0, np.exp(p[..., hd] - p[..., hd].max(0)), 0)
    ref = (np.einsum('sh,shc->hc', e, p[..., :hd]) / (e * p[..., hd + 1]).sum(0)[:, None]).ravel()
    for flags in (CFG_DYNAMIC, CFG_STATIC):
        with Executor(flags=flags) as ex:
            ex.load(b)
            ex.run()
            assert np.abs(ex.read_buffer('o')[0] - ref).max() <= 2.0 ** -23 * (S + 4) * np.abs(ref).max()
