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
