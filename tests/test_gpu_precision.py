"""Distances of the streamed and reduced-order kernel forms from float64 evaluations of the same op on the same stored inputs.  Bounds follow
from the storage type (half a unit of bf16) or from the number of float32 roundings on the path; none is a measured value."""
import numpy as np
import pytest

from kvm_b200.executor import Executor
from kvm_b200.workloads.graph import Graph
from oracle.ops_np import bf16_round

pytestmark = pytest.mark.gpu


def run(g):
    ex = Executor()
    ex.load(g.to_bundle())
    ex.run()
    return ex


def gemv_task(g, op, x, w, out, n0, n1, K, pro=0, x2=None, gamma=None):
    rows = {'r0': 0, 'r1': 1} if op == 'gemv_bf16_rows' else {}
    g.task(op, {'x': x, 'x2': x2, 'gamma': gamma, 'w': w, 'out': out, 'res': None, 'n0': n0, 'n1': n1, 'K': K, 'pro': pro, 'eps': 1e-6, **rows}, [x], [(out, (0, 1), (n0, n1))])


@pytest.mark.parametrize('op,K', [('gemv_bf16', 1024), ('gemv_bf16', 4864), ('gemv_bf16', 12296), ('gemv_bf16_rows', 1024)])
def test_swiglu_activations_are_the_rounded_values(kvm_lib, op, K):
    # weight row n picks one activation alone: the output is bf16(silu(x) * x2), far tails included (silu(-87) is a normal float32)
    x = np.concatenate([np.linspace(-95, 95, K // 2), np.random.default_rng(1).standard_normal(K // 2) * 3]).astype(np.float32)
    pick = np.linspace(0, K - 1, 512).astype(int)
    w = np.zeros((512, K), np.float32)
    w[np.arange(512), pick] = 1
    g = Graph('silu')
    g.data('x', x[None]), g.data('u', np.full((1, K), 1.5, np.float32)), g.data('w', w, 'bf16'), g.buffer('o', 1, 512)
    for n in range(0, 512, 64):
        gemv_task(g, op, 'x', 'w', 'o', n, n + 64, K, pro=2, x2='u')
    ex = run(g)
    assert ex.plan_info()[:2] == (True, True)
    x = x[pick].astype(np.float64)
    ref = 1.5 * x / (1 + np.exp(-x))
    got = ex.read_buffer('o')[0].astype(np.float64)
    # half a unit of bf16 (normal and subnormal), and the float32 evaluation's few units on top
    assert (np.abs(got - ref) <= 2.0 ** -8 * (1 + 2.0 ** -10) * np.abs(ref) + 2.0 ** -134).all()
    ex.close()


def lse_bias(got, ref):
    """Mean signed error in units of the float32 spacing at the references' size."""
    return float((got - ref).mean() / np.spacing(np.abs(ref).mean().astype(np.float32)))


@pytest.mark.parametrize('T,hd', [(300, 128), (200, 64), (130, 32)])
def test_attention_scores_do_not_drift(kvm_lib, T, hd):
    # Products of one sign: a sum kept in the matrix unit's accumulator loses part of a unit with every instruction.  Sixteen products
    # added from zero lose half a unit of their own sum on average, which is 16 / hd of the score: half a unit of the score altogether;
    # the float32 adds between them round to nearest, without a mean.
    rng = np.random.default_rng(0)
    q, k = (bf16_round(np.abs(rng.standard_normal((T, hd)) * 3).astype(np.float32)) for _ in range(2))
    g = Graph('attn')
    g.data('q', q, 'bf16'), g.data('k', k, 'bf16'), g.data('v', k, 'bf16'), g.buffer('o', T, hd), g.buffer('lse', T, 1)
    for q0 in range(0, T, 128):
        q1 = min(q0 + 128, T)
        g.task('attn_fwd', {'q': 'q', 'k': 'k', 'v': 'v', 'o': 'o', 'lse': 'lse', 'b': 0, 'h': 0, 'q0': q0, 'T': T, 'H': 1, 'Hkv': 1, 'hd': hd, 'scale': hd ** -0.5},
               ['q'], [('o', (q0, q1), (0, hd)), ('lse', (q0, q1))])
    ex = run(g)
    assert ex.tc_task_count() == 0
    s = q.astype(np.float64) @ k.astype(np.float64).T * np.float64(np.float32(hd ** -0.5))
    s[np.triu_indices(T, 1)] = -np.inf
    m = s.max(1, keepdims=True)
    ref = (m + np.log(np.exp(s - m).sum(1, keepdims=True)))[:, 0]
    assert abs(lse_bias(ex.read_buffer('lse')[:, 0], ref)) <= 0.5
    ex.close()


@pytest.mark.parametrize('hd,G', [(128, 4), (128, 8), (64, 7), (32, 8)])
def test_split_scores_do_not_drift(kvm_lib, hd, G):
    # The same for the split decode attention.  Queries are rotated back from positive bf16 values, which the kernel's rotation and
    # rounding restore exactly.
    rng = np.random.default_rng(0)
    n, S, theta, half = 1000, 8, 1e4, hd // 2
    pos, keys = bf16_round(np.abs(rng.standard_normal((G, hd)) * 3).astype(np.float32)), bf16_round(np.abs(rng.standard_normal((n, hd)) * 3).astype(np.float32))
    ang = np.float64(n - 1) * np.float32(theta ** (-2.0 * np.arange(half) / hd)).astype(np.float64)
    a, b = pos[:, :half].astype(np.float64), pos[:, half:].astype(np.float64)
    q = np.concatenate([a * np.cos(ang) + b * np.sin(ang), b * np.cos(ang) - a * np.sin(ang)], 1).astype(np.float32)
    g = Graph('part')
    g.data('q', q.reshape(1, -1)), g.data('kc', keys, 'bf16'), g.data('vc', keys, 'bf16'), g.data('lens', np.array([[n - 1]], np.int32), 'i32'), g.buffer('part', S * G, hd + 2)
    g.buffer('new', 1, hd)
    for s in range(S):
        g.task('attn_decode_part', {'q': 'q', 'kc': 'kc', 'vc': 'vc', 'lens': 'lens', 'part': 'part', 'knew': 'new', 'vnew': 'new', 'b': 0, 'kvh': 0, 's': s, 'S': S, 'H': G, 'Hkv': 1,
                                    'hd': hd, 'Tmax': n, 'scale': hd ** -0.5, 'theta': theta, 'flags': 3}, ['q'], [('part', (s * G, s * G + G))])
    g.buffer('w', 8, 256, 'bf16'), g.buffer('x', 1, 256), g.buffer('y', 1, 8)
    gemv_task(g, 'gemv_bf16', 'x', 'w', 'y', 0, 8, 256)          # a program with a streamed GEMV runs on the static path, its splits from the ring
    ex = run(g)
    assert ex.plan_info()[:2] == (True, True)
    keys[n - 1] = 0                                               # the appended key
    s = pos.astype(np.float64) @ keys.astype(np.float64).T * np.float64(np.float32(hd ** -0.5))
    s = s.reshape(G, S, n // S)
    m = s.max(2)
    ref = (m + np.log(np.exp(s - m[..., None]).sum(2))).T
    part = ex.read_buffer('part').reshape(S, G, hd + 2).astype(np.float64)
    assert abs(lse_bias(part[..., hd] + np.log(part[..., hd + 1]), ref)) <= 0.5
    ex.close()


def test_gemv_sums_in_pairs(kvm_lib):
    # Terms of random sign: an addition in which partial sums of all terms meet adds (c * sum)^2 to the error's variance, c = 0.41 * 2^-24
    # the rms of a rounding relative to the rounded value.  A row of 4096 passes a chain of four products (2.5 such levels on average),
    # the halves of a packed sum (1), five shuffles and sixteen parts in pairs (4).  Parts one after the other would count 8.5.
    K, levels = 4096, 2.5 + 1 + 5 + 4
    rng = np.random.default_rng(1)
    x, w = bf16_round(rng.standard_normal(K).astype(np.float32)), bf16_round((rng.standard_normal((512, K)) * 0.02).astype(np.float32))
    g = Graph('gemv')
    g.data('x', x[None]), g.data('w', w, 'bf16'), g.buffer('o', 1, 512)
    for n in range(0, 512, 64):
        gemv_task(g, 'gemv_bf16', 'x', 'w', 'o', n, n + 64, K)
    ex = run(g)
    ref = w.astype(np.float64) @ x.astype(np.float64)
    assert np.linalg.norm(ex.read_buffer('o')[0] - ref) <= 0.41 * 2.0 ** -24 * levels ** 0.5 * np.linalg.norm(ref)
    ex.close()


@pytest.mark.parametrize('T,hd', [(200, 32), (257, 64)])
def test_attention_gradients_do_not_shrink(kvm_lib, T, hd):
    # dq of float32 inputs: scores, their gradient and the weighted sum of the keys each lose half a unit (2^-25 to 2^-24) of their sum
    # on average where the products of the leading terms are added; every other addition is rounded to nearest.  Projected on the result
    # the roundings average out and the losses add up: at most 2^-23.
    rng = np.random.default_rng(0)
    q, k, v, do = (rng.standard_normal((T, hd)).astype(np.float32) for _ in range(4))
    Q, K, V, D = (a.astype(np.float64) for a in (q, k, v, do))
    sc = np.float64(np.float32(hd ** -0.5))
    s = Q @ K.T * sc
    s[np.triu_indices(T, 1)] = -np.inf
    m = s.max(1, keepdims=True)
    lse = (m + np.log(np.exp(s - m).sum(1, keepdims=True))).astype(np.float32)
    delta = ((np.exp(s - lse.astype(np.float64)) @ V) * D).sum(1, keepdims=True).astype(np.float32)
    dS = np.exp(s - lse.astype(np.float64)) * (D @ V.T - delta.astype(np.float64))
    g = Graph('attn')
    for n, a in (('q', q), ('k', k), ('v', v), ('do', do), ('lse', lse), ('delta', delta)):
        g.data(n, a)
    g.buffer('dq', T, hd), g.buffer('dk', T, hd), g.buffer('dv', T, hd)
    for r0 in range(0, T, 128):
        r1, args = min(r0 + 128, T), {'q': 'q', 'k': 'k', 'v': 'v', 'do': 'do', 'lse': 'lse', 'delta': 'delta', 'b': 0, 'T': T, 'H': 1, 'hd': hd, 'scale': hd ** -0.5}
        g.task('attn_bwd_dq', {**args, 'dq': 'dq', 'h': 0, 'q0': r0, 'Hkv': 1}, ['q'], [('dq', (r0, r1), (0, hd))])
        g.task('attn_bwd_dkv', {**args, 'dk': 'dk', 'dv': 'dv', 'kvh': 0, 'k0': r0}, ['q'], [('dk', (r0, r1), (0, hd)), ('dv', (r0, r1), (0, hd))])
    ex = run(g)
    for name, ref in (('dq', dS @ K * sc), ('dk', dS.T @ Q * sc)):
        assert abs(((ex.read_buffer(name) - ref) * ref).sum() / (ref * ref).sum()) <= 2.0 ** -23, name
    ex.close()
