"""The work that users have this framework do, as cases that can be timed: one launch (or a short run of launches) of a compiled
program through the executor's public entry points, over the sizes in use.

Three families, each a program of the workload generators:
  train    decoder-only language model, forward + backward + clip + AdamW, f32 or bf16 storage, `steps` optimizer steps a launch
  mlp      several MLP classifiers trained side by side in one launch, f32, SGD with momentum
  decode   greedy generation of `tokens` tokens per request from a filled KV cache, the requests as rows of one batch or as
           independent users

A program keeps its weights, optimizer state and caches in a few torch tensors ("arenas") whose slices are bound as the program's
buffers, as a PyTorch host does; everything else is allocated by the executor.  A pass re-runs the resident program: training
goes on from the weights it has, on the next window of the token stream; decode starts again from the end of the prompt.
"""
from __future__ import annotations

import functools
import math

import torch

from kvm_b200.executor import Executor
from kvm_b200.workloads.decode import DecodeConfig, build_decode, build_decode_rows
from kvm_b200.workloads.gpt import GPTConfig, build_training
from kvm_b200.workloads.mlp import MLPConfig, build_mlps

TORCH_TYPE = {0: torch.float32, 1: torch.int32, 2: torch.bfloat16}
ALIGN = 64                # elements: slices of an arena start on 128-byte boundaries at least
WINDOWS = 256             # training windows in the token stream before it starts over


def train(name, precision, layers, d_model, heads, d_ff, vocab, seq, batch, steps=1, tied=False):
    return dict(name=name, family='train', precision=precision, layers=layers, d_model=d_model, heads=heads, d_ff=d_ff, vocab=vocab, seq=seq, batch=batch,
                steps=steps, tied=tied)


def mlp(name, widths, in_dim, classes, batch, steps=1):
    return dict(name=name, family='mlp', widths=' '.join(map(str, widths)), in_dim=in_dim, classes=classes, batch=batch, steps=steps)


def decode(name, layers, hidden, heads, kv_heads, head_dim, ffn, vocab, ctx, batch=1, rows=False, qk_norm=False, tokens=1):
    return dict(name=name, family='decode', layers=layers, hidden=hidden, heads=heads, kv_heads=kv_heads, head_dim=head_dim, ffn=ffn, vocab=vocab, ctx=ctx,
                batch=batch, rows=rows, qk_norm=qk_norm, tokens=tokens)


def listed():
    return [
        # The tiny training graph (config 1): one launch a step, as a loop that looks at the loss after each step runs it.
        train('train_tiny_f32', 'f32', 2, 128, 4, 512, 256, 64, 8, tied=True),
        # A small f32 model of odd sizes, several steps in one launch (experiments that read the loss back now and then).
        train('train_small_f32_4steps', 'f32', 3, 192, 3, 768, 1001, 120, 5, steps=4),
        # bf16 storage at a batch that fills no whole tile: 3 sequences of 200 tokens, heads of 128.
        train('train_ragged_bf16', 'bf16', 3, 640, 5, 2560, 5000, 200, 3),
        # The widths of the 355M model (config 4), two of its layers.
        train('train_355m_2layers_bf16', 'bf16', 2, 1024, 16, 4096, 50304, 1024, 8),
        # The 162M model (config 3), micro-batch 8 x 1024: the headline step.
        train('train_162m_bf16', 'bf16', 12, 768, 12, 3072, 50304, 1024, 8),
        # Hyper-parameter searches: a few small networks of odd widths, several steps a launch ...
        mlp('mlp_small_4steps', (72, 104, 200), 100, 10, 96, steps=4),
        # ... and the eight widths of config 2.
        mlp('mlp_8_widths', (128, 256, 384, 512, 768, 1024, 1536, 2048), 512, 10, 256),
        # One short request on a tiny model: the latency of a token.
        decode('decode_tiny', 2, 256, 8, 2, 32, 512, 1000, 40, tokens=4),
        # A small model of the sizes such models have (hidden 896, seven query heads per key head), one user.
        decode('decode_small', 12, 896, 14, 2, 64, 4864, 32000, 700, tokens=2),
        # Three users with a program each in one launch, QK norm.
        decode('decode_users3_qknorm', 8, 1024, 16, 8, 128, 3072, 50304, 1500, batch=3, qk_norm=True, tokens=2),
        # The 8B shape (config 5) for one user at 4K context.
        decode('decode_8b', 36, 4096, 32, 8, 128, 12288, 151936, 4096),
        # Eight users as rows of one batch, four layers of the 8B shape.
        decode('decode_8b_4layers_rows8', 4, 4096, 32, 8, 128, 12288, 151936, 4096, batch=8, rows=True, tokens=2),
    ]


def log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step) * step))


def draw(rng):
    while True:
        family = rng.choice(('train f32', 'train bf16', 'train bf16', 'mlp', 'decode', 'decode', 'decode'))
        if family == 'train f32':
            hd = rng.choice((32, 64))
            heads = rng.randint(1, 256 // hd)
            c = train('', 'f32', rng.randint(1, 4), heads * hd, heads, heads * hd * rng.choice((2, 4)), log_int(rng, 65, 2000), log_int(rng, 16, 256), rng.randint(1, 9),
                      rng.randint(1, 4), rng.random() < 0.5)
            top = 2e10
        elif family == 'train bf16':
            hd = rng.choice((64, 64, 128))
            heads = rng.randint(2, 1024 // hd)
            c = train('', 'bf16', rng.randint(1, 6), heads * hd, heads, heads * hd * 4, log_int(rng, 1000, 50304, 8), log_int(rng, 64, 1024 if hd == 64 else 384),
                      rng.randint(1, 8))
            top = 4e12
        elif family == 'mlp':
            c = mlp('', [log_int(rng, 48, 2048) for _ in range(rng.randint(1, 8))], log_int(rng, 64, 1024), log_int(rng, 10, 200), log_int(rng, 32, 512), rng.randint(1, 4))
            top = 4e10
        else:
            hd, group = rng.choice((64, 128)), rng.choice((1, 2, 4, 4, 7, 8))
            kv = rng.randint(1, 8)
            rows = rng.random() < 0.4
            c = decode('', rng.randint(2, 16), log_int(rng, 256, 4096, 128), group * kv, kv, hd, log_int(rng, 512, 12288, 128), log_int(rng, 1000, 151936), log_int(rng, 16, 4096),
                       rng.randint(2, 8) if rows else rng.choice((1, 1, 1, 2, 4)), rows, rng.random() < 0.3, rng.randint(1, 4))
            top = 5e9
        w = work(c)
        # no more than the largest listed cases cost, and a program that is compiled in a few seconds
        if (w['bytes'] if c['family'] == 'decode' else w['flops']) <= top and task_estimate(c) <= 40000:
            del c['name']
            return c


def task_estimate(c):
    """Tasks of the case's program, roughly."""
    if c['family'] == 'train':
        tokens, d, f, tm, tn = c['batch'] * c['seq'], c['d_model'], c['d_ff'], *((128, 256) if c['precision'] == 'bf16' else (64, 64))
        tiles = lambda m, n: -(-m // tm) * -(-n // tn)
        layer = 8 * tiles(tokens, d) + 4 * tiles(d, d) + 2 * tiles(tokens, f) + tiles(d, f) + tiles(f, d) + 3 * c['batch'] * c['heads'] * -(-c['seq'] // 128) + tokens // 4
        return c['steps'] * (c['layers'] * layer + 3 * tiles(tokens, c['vocab']) + tokens // 8)
    if c['family'] == 'mlp':
        return c['steps'] * sum(3 * (-w // 64) ** 2 + 6 * (-w // 64) * (-c['batch'] // 64) for w in widths(c))
    users = 1 if c['rows'] else c['batch']
    return c['layers'] * (users * 900 + c['batch'] * c['kv_heads'] * (splits(c) + 1))


def widths(c):
    return [int(w) for w in c['widths'].split()]


def splits(c):
    """Context splits of the decode attention: one wave of tasks over the SMs, 64 keys or more in each."""
    return max(1, min(136 // c['kv_heads'], -(-c['ctx'] // 64), 17))


def matmul_params(c):
    """Elements of the weight matrices that one pass multiplies with."""
    if c['family'] == 'train':
        d = c['d_model']
        return c['layers'] * (4 * d * d + 2 * d * c['d_ff']) + c['vocab'] * d
    if c['family'] == 'mlp':
        return sum(c['in_dim'] * w + w * w + w * c['classes'] for w in widths(c))
    h, q, kv = c['hidden'], c['heads'] * c['head_dim'], c['kv_heads'] * c['head_dim']
    return c['layers'] * (2 * h * q + 2 * h * kv + 3 * h * c['ffn']) + c['vocab'] * h


def work(c):
    m = matmul_params(c)
    if c['family'] == 'train':
        tokens = c['batch'] * c['seq']
        params = m + (0 if c['tied'] else c['vocab'] * c['d_model']) + c['seq'] * c['d_model']
        attention = 3.5 * c['layers'] * 2 * c['batch'] * c['seq'] ** 2 * c['d_model']          # causal: half of the score matrix
        # per parameter: weight and two moments read and written, gradient written
        return {'flops': c['steps'] * (6.0 * m * tokens + attention), 'bytes': c['steps'] * (28.0 * params + 8.0 * tokens)}
    if c['family'] == 'mlp':
        return {'flops': c['steps'] * 6.0 * m * c['batch'], 'bytes': c['steps'] * (20.0 * m + 4.0 * c['batch'] * c['in_dim'])}
    kv = c['layers'] * 2 * c['batch'] * c['kv_heads'] * c['ctx'] * c['head_dim']
    return {'bytes': c['tokens'] * (2.0 * m + 2.0 * kv + 4.0 * c['batch'] * c['vocab']),
            'flops': c['tokens'] * (2.0 * m * c['batch'] + 2.0 * kv * (c['heads'] // c['kv_heads']))}


def tolerance(c):
    # f32 programs: sums of a few thousand f32 terms, carried through one to four AdamW or momentum steps.  bf16 storage: eight bits.
    return {'rel': 1e-4} if c['family'] == 'mlp' or (c['family'] == 'train' and c['precision'] == 'f32') else {'rel': 1e-2}


def config(c):
    if c['family'] == 'train':
        flat = 262144 if c['precision'] == 'bf16' else 65536
        rows = (64 if c['batch'] * c['seq'] >= 4096 else 16) if c['precision'] == 'bf16' else 16
        return GPTConfig(layers=c['layers'], d_model=c['d_model'], heads=c['heads'], d_ff=c['d_ff'], vocab=c['vocab'], seq=c['seq'], batch=c['batch'], tied=c['tied'],
                         precision=c['precision'], flat_chunk=flat, norm_rows=rows)
    if c['family'] == 'mlp':
        return MLPConfig(widths=tuple(widths(c)), in_dim=c['in_dim'], classes=c['classes'], batch=c['batch'])
    return DecodeConfig(layers=c['layers'], hidden=c['hidden'], heads=c['heads'], kv_heads=c['kv_heads'], head_dim=c['head_dim'], ffn=c['ffn'], vocab=c['vocab'], ctx=c['ctx'],
                        tmax=c['ctx'] + 64, batch=c['batch'], splits=splits(c), qk_norm=c['qk_norm'], rows_per_task=0, join_threshold=1000)


@functools.lru_cache(maxsize=2)
def compiled(key):
    """The case's program, compiled once; the inputs of a pass are data of the program, not part of it."""
    c = dict(key)
    cfg = config(c)
    if c['family'] == 'train':
        g = build_training(cfg, c['steps'], stream_steps=WINDOWS * c['steps'])
    elif c['family'] == 'mlp':
        g = build_mlps(cfg, c['steps'])
    else:
        g = (build_decode_rows if c['rows'] else build_decode)(cfg)
    return g.to_bundle(check=False)


def arena_of(family, name):
    """The tensor that buffer `name` is a slice of; None for what the program keeps to itself."""
    last = name.split('.')
    if family == 'train':
        if last[0] in ('w', 'm', 'v', 'g', 'loss'):
            return last[0]
        return name if name in ('stream_ids', 'stream_tgt', 'opt_step') else None
    if family == 'mlp':
        if last[0] in 'xy':
            return last[0]
        return last[1] if last[1] in ('g', 'v', 'loss') else 'w' if last[1] in ('w1', 'b1', 'w2', 'b2', 'w3', 'b3') else None
    if last[0] == 'wb':
        return 'w'
    return {'kc': 'kv', 'vc': 'kv', 'lens': 'request', 'tok': 'request', 'logits': 'logits'}.get(last[-1])


def fill(t, init, gen):
    """Values of the distribution a buffer's `init` names, from this seed's generator."""
    if init['kind'] == 'fill':
        if init['value']:
            t.fill_(init['value'])
    elif init['kind'] == 'seeded' and init['draws'] == 1:
        t.uniform_(-init['bias'] * init['coef'], (1 - init['bias']) * init['coef'], generator=gen)
    elif init['kind'] == 'seeded':
        t.normal_(0.0, init['coef'] / math.sqrt(3.0), generator=gen)      # the seeded normal adds four uniform draws


def prepare(case, seed):
    family = case['family']
    bundle = compiled(tuple(sorted((k, v) for k, v in case.items() if k != 'name')))
    gen = torch.Generator('cuda').manual_seed(seed)
    ex = Executor()
    ex.set_stream(torch.cuda.current_stream().cuda_stream)
    size, kind, place = {}, {}, {}
    for b in bundle.buffers:
        if key := arena_of(family, b['name']):
            place[b['name']] = size.get(key, 0)
            size[key] = place[b['name']] + -(-b['rows'] * b['cols'] // ALIGN) * ALIGN
            kind[key] = TORCH_TYPE[b['dtype']]
    arena = {k: torch.zeros(n, dtype=kind[k], device='cuda') for k, n in size.items()}
    view = {}
    for b in bundle.buffers:
        name = b['name']
        if key := arena_of(family, name):
            at = place[name]
            view[name] = arena[key][at:at + b['rows'] * b['cols']].view(b['rows'], b['cols'])
            fill(view[name], b['init'], gen)
            ex.bind_buffer(view[name].data_ptr(), b['rows'], b['cols'], b['dtype'], name=name)
        else:
            ex.add_bundle_buffer(bundle, b)
    ex.submit(bundle.tasks, bundle.succ, bundle.args)
    state = {'case': case, 'ex': ex, 'arena': arena}
    if family == 'train':
        n = case['batch'] * case['seq']
        tokens = torch.randint(case['vocab'], (WINDOWS * case['steps'], case['batch'], case['seq'] + 1), dtype=torch.int32, device='cuda', generator=gen)
        view['stream_ids'].view(-1, n).copy_(tokens[:, :, :-1].reshape(-1, n))
        view['stream_tgt'].view(-1, n).copy_(tokens[:, :, 1:].reshape(-1, n))
        state['windows'] = WINDOWS
    elif family == 'mlp':
        for s in range(case['steps']):
            view[f'y.{s}'].random_(0, case['classes'], generator=gen)
    else:
        # A trained model is sure of most of its tokens: embedding rows that stand out of the residual stream and a head whose
        # row for the next token lies along the current one's embedding give such peaked distributions.
        view['wb.embed'].normal_(0.0, 4.0, generator=gen)
        view['wb.head'].copy_(torch.roll(view['wb.embed'], 1, 0).mul_(0.02 / 4.0))
        for name, t in view.items():
            if name.endswith('lens'):
                t.fill_(case['ctx'])
            elif name.endswith('tok'):
                t.random_(0, case['vocab'], generator=gen)
        state['prompt'] = arena['request'].clone()
    return state


def run(state):
    case, ex, arena = state['case'], state['ex'], state['arena']
    if case['family'] == 'decode':
        arena['request'].copy_(state['prompt'])                # the end of the prompt: last token, tokens in the cache
        ex.run_steps(case['tokens'])
        return {k: arena[k] for k in ('request', 'logits', 'kv')}
    if case['family'] == 'train':
        if state['windows'] == 0:                              # the stream is used up: from its start again
            arena['opt_step'].zero_()
            state['windows'] = WINDOWS
        state['windows'] -= 1
    ex.run()
    return {k: arena[k] for k in ('loss', 'w', 'm', 'v', 'g') if k in arena}
