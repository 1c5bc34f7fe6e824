"""The form of latent attention that up-projects a portion's context: which sizes and steps take it (CPU), and layers with
heads of 64 and 128 through the engine against the plain implementations."""

import json
from types import SimpleNamespace

import pytest
import torch

from edgerag_b200.ops import kernels


@pytest.mark.parametrize("rank", [8, 64, 512, 520, 576, 640, 960, 1024])
@pytest.mark.parametrize("dim,rot,v", [(64, 8, 64), (64, 32, 128), (128, 64, 128), (128, 64, 64)])
def test_no_size_is_rounded_more_than_in_the_latent_space(dim, rot, v, rank):
    """Where the latent space has float32 queries and weights (the general kernel), the up-projected form is not taken."""
    wide = kernels.latent_wide_supported(torch.bfloat16, dim, rot, v, rank)
    assert wide == (kernels.latent_mma_supported(torch.bfloat16, rank, rot) and rank <= 512)
    assert not kernels.latent_wide_supported(torch.float32, dim, rot, v, rank)


def _mixer(heads, dim, rot, v, rank, **more):
    from edgerag_b200.parts.latent_attention import LatentAttention

    return LatentAttention(64, heads, dim, rot, v, rank, 0.1, 10000.0, rot, 1e-5, torch.bfloat16, torch.device("cpu"), **more)


@pytest.mark.parametrize("mixer,lens,rows,wide", [
    # device times of the sublayer, up-projected | in the latent space
    ((16, 128, 64, 128, 512), [2], 64, True),                         # 25 | 35 us
    ((16, 128, 64, 128, 512), [2], 8192, True),                       # 204 | 645
    ((16, 128, 64, 128, 512), [2, 3, 3, 3], 8192, True),              # 285 | 646
    ((16, 128, 64, 128, 512), [2] * 8, 2048, True),                   # 125 | 189
    ((16, 128, 64, 128, 512), [2] * 16, 2048, False),                 # 187 to 232 | 189 to 191
    ((16, 128, 64, 128, 512), [2] * 16, 512, False),                  # 96 | 74
    ((16, 128, 64, 128, 512), [2] * 32, 1024, False),                 # 186 | 113
    ((16, 128, 64, 128, 512), [2] * 32, 64, False),                   # 62 | 41
    ((16, 128, 64, 128, 512), [512] + [17] * 15, 2048, True),         # 205 | 350
    ((16, 128, 64, 128, 512), [512] + [17] * 15, 512, True),          # 99 | 119
    ((16, 128, 64, 128, 512), [1531, 517], 1536, True),
    ((8, 64, 32, 64, 256), [2], 64, True),                            # 21 | 23
    ((8, 64, 32, 64, 256), [2] * 16, 2048, True),                     # 74 | 133
    ((8, 64, 32, 64, 256), [2] * 32, 64, False),                      # 34 | 29
])
def test_portions_take_the_faster_form(mixer, lens, rows, wide, monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    step = SimpleNamespace(batch_invariant=False, host_q_len=lens, n_decode=0, max_keys_bound=lambda: rows)
    assert _mixer(*mixer)._wide_rows(step) == (rows if wide else 0)
    # beside single tokens whose contexts set the bound, and where nothing may depend on the step: the latent space
    step.host_q_len, step.n_decode = [1] * 8 + lens, 8
    if rows * len(lens) > 32 * sum(lens) + 2048:
        assert _mixer(*mixer)._wide_rows(step) == 0
    step.batch_invariant = True
    assert _mixer(*mixer)._wide_rows(step) == 0


def test_rows_follow_the_window_and_the_limit_of_bytes(monkeypatch):
    monkeypatch.setattr(kernels, "_sms", lambda device: 148)
    step = SimpleNamespace(batch_invariant=False, host_q_len=[100], n_decode=0, max_keys_bound=lambda: 4096)
    mixer = _mixer(16, 128, 64, 128, 512, window=200)
    assert mixer._wide_rows(step) == 384                              # 200 + 100 + 63 keys, whole tiles of 64
    mixer.WIDE_MAX_BYTES = 2 * 384 * 16 * 256 - 1
    assert mixer._wide_rows(step) == 0


def test_scratch_grows_seldom_while_a_prompt_is_read():
    """Portions of 512 tokens up to a context of 32,768, whose bounds are quarters of a power of two: seven sizes, all within the limit."""
    mixer = _mixer(16, 128, 64, 128, 512)
    most = mixer.WIDE_MAX_BYTES // (2 * 16 * 256)
    bounds = [kernels.context_bound(past // 16)[0] * 16 for past in range(512, 32769, 512)]
    rooms = [mixer._wide_room(rows) for rows in bounds]
    assert all(rows <= room <= most for rows, room in zip(bounds, rooms)) and len(set(rooms)) == 7 < len(set(bounds))
    assert mixer._wide_room(most - 64) == most and mixer._wide_room(64) == 64


# --- through the engine ------------------------------------------------------------------------------------------------

def _models():
    import plain_dokodra
    import plain_pudadra
    import plain_sabolorn

    pud, sab = plain_pudadra, plain_sabolorn
    att = lambda kind, m, **more: {"type": kind, "mixer": {**m, **more}, "mlp": None}      # noqa: E731
    gated = {"heads": 3, "dim": 64, "rot_dim": 16, "vdim": 128, "kv_rank": 48, "scale": 0.1, "rot": {"base": 900.0, "dims": 16}}
    sinks = {"heads": 2, "dim": 128, "rot_dim": 64, "vdim": 64, "kv_rank": 72, "q_rank": 40, "scale": 0.08, "rot": {"base": 20000.0, "dims": 64}}
    source = sab.latent_layer(heads=2, dim=64, rot_dim=32, vdim=64, kv_rank=64, q_rank=24, mlp=sab.dense_mlp(40),
                              scaling={"factor": 6.0, "original": 64, "fast": 8.0, "slow": 1.0})
    reader = {**source, "mixer": {**source["mixer"], "heads": 3, "dim": 128, "vdim": 128, "kv_from": 0}}
    return {
        # a gate per head, a second layer that reads the first one's rows, and sinks behind queries with a latent of their own
        "gates_sinks": ({"architecture": "Dokodra", "width": 88, "vocab": 211, "embedding": {"scale": 1.7}, "norm": {"eps": 1e-6}, "logit_softcap": 12.0,
                         "layers": [att("latent_attention", gated), att("latent_attention", gated, kv_from=0), att("latent_attention_2", sinks)]},
                        plain_dokodra.random_tensors, lambda w, raw, tokens: plain_dokodra.forward(raw, w, tokens)),
        # windows shorter and longer than a tile of 64 keys, and none; no gates
        "windows": (pud.make_config([pud.latent_layer(heads=3, dim=64, rot_dim=32, vdim=64, kv_rank=40, window=27, mlp=pud.dense_mlp(40)),
                                     pud.latent_layer(heads=2, dim=128, rot_dim=64, vdim=128, kv_rank=96, window=100, mlp=pud.dense_mlp(48)),
                                     pud.latent_layer(heads=4, dim=64, rot_dim=8, vdim=128, kv_rank=64, window=0, mlp=None)], width=80, vocab=203),
                    pud.random_weights, pud.forward),
        # a gate per entry, stretched rotations, another layer's cache
        "entry_gates": (sab.make_config([source, reader], width=72, vocab=61, side=0, softcap=0.0), sab.random_weights, sab.forward),
    }


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    from edgerag_b200.weights.safetensors_io import write_safetensors

    made = {}

    def get(name):
        if name not in made:
            raw, weights, forward = _models()[name]
            folder, tensors = tmp_path_factory.mktemp(name), weights(raw, 0)
            (folder / "config.json").write_text(json.dumps(raw))
            write_safetensors(folder / "model.safetensors", tensors)
            made[name] = (folder, raw, lambda tokens: forward(tensors, raw, tokens))
        return made[name]

    return get


@pytest.fixture
def calls(monkeypatch):
    """Every layer's portions take the up-projected form where it can; the kernel's calls are counted."""
    from edgerag_b200.parts.latent_attention import LatentAttention

    count, kernel = [], kernels.latent_attention_wide
    monkeypatch.setattr(LatentAttention, "_wide_pays", lambda self, lens, rows: True)
    monkeypatch.setattr(kernels, "latent_attention_wide", lambda *a, **k: (count.append(a[0].shape[0]), kernel(*a, **k)))
    return count


def _engine(folder, **over):
    from edgerag_b200.engine.engine import Engine, EngineOptions

    opts = dict(dtype="bfloat16", block_size=16, num_blocks=96, max_batch_size=4, max_step_tokens=1024, max_model_len=1 << 20, cuda_graphs=False,
                poison_freed_pages=True)
    return Engine.from_pretrained(folder, EngineOptions(**{**opts, **over}))


def _tokens(raw, n, seed):
    return torch.randint(0, raw["vocab"], (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _close(got, want, what):
    """Logits of a bfloat16 engine against float64 (activations are rounded to 8 bits between the products): the bands of the other models'
    tests, 2.5e-2 of a row's spread on average and 0.12 at worst; a lost key or a wrong head moves a row by more."""
    assert torch.isfinite(got).all(), what
    d, w = got.double() - want.double(), want.double() - want.double().mean(-1, keepdim=True)
    d = d - d.mean(-1, keepdim=True)
    e = d.pow(2).mean(-1).sqrt() / w.pow(2).mean(-1).sqrt().clamp_min(1e-9)
    assert e.mean() < 2.5e-2 and e.max() < 0.12, (what, e.mean().item(), e.max().item())


def _feed(runner, rid, tokens, cuts):
    from edgerag_b200.engine.step import StepEntry

    rows, at = [], 0
    for n in cuts:
        rows.append(runner.step([StepEntry(rid, tokens=tokens[at: at + n], want=list(range(n)))]).float().cpu().clone())
        at += n
    assert at == len(tokens)
    return torch.cat(rows)


NAMES = ["gates_sinks", "windows", "entry_gates"]


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_portions_of_a_prompt_through_the_engine(name, model, calls):
    folder, raw, forward = model(name)
    engine = _engine(folder)
    tokens = _tokens(raw, 300, 1)
    want = forward(tokens)
    for cuts in ([300], [64, 2, 1, 1, 130, 63, 1, 38], [3, 257, 40]):
        calls.clear()
        engine.runner.admit(0)
        _close(_feed(engine.runner, 0, tokens, cuts), want, (name, cuts))
        engine.runner.release(0)
        assert len(calls) == len(raw["layers"]) * sum(n > 1 for n in cuts)
    assert int(engine.runner.status) == 0
    engine.cache.check_invariants()


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_portions_beside_single_tokens(name, model, calls):
    """A step of two single tokens and two portions: the former in the latent space, the latter up-projected, each its own rows."""
    from edgerag_b200.engine.step import StepEntry

    folder, raw, forward = model(name)
    engine = _engine(folder)
    tokens = [_tokens(raw, n, 10 + i) for i, n in enumerate((71, 140, 97, 210))]
    got = [[] for _ in tokens]
    for r in range(4):
        engine.runner.admit(r)

    def step(parts):
        entries = [StepEntry(r, tokens=tokens[r][a:b], want=list(range(b - a))) for r, a, b in parts]
        out, at = engine.runner.step(entries).float().cpu(), 0
        for r, a, b in parts:
            got[r].append(out[at: at + b - a].clone())
            at += b - a

    step([(0, 0, 70), (1, 0, 139), (2, 0, 30)])
    calls.clear()
    step([(3, 0, 150), (0, 70, 71), (2, 30, 97), (1, 139, 140)])
    assert len(calls) == len(raw["layers"]) and set(calls) == {219}
    step([(3, 150, 210)])
    for r, t in enumerate(tokens):
        _close(torch.cat(got[r]), forward(t), (name, r))
    assert int(engine.runner.status) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAMES)
def test_a_replayed_step_reads_its_own_request(name, model, calls):
    """The same cuts for three requests: eager, captured and replayed, over other tokens, pages and (the last) another past."""
    folder, raw, forward = model(name)
    engine = _engine(folder, cuda_graphs=True)
    for r in range(4):
        tokens = _tokens(raw, 190 if r < 3 else 176, 20 + r)
        cuts = [100, 60, 30] if r < 3 else [86, 60, 30]
        engine.runner.admit(r)
        _close(_feed(engine.runner, r, tokens, cuts), forward(tokens), (name, r))
        if r != 1:                                      # (one stays: the next request has other pages)
            engine.runner.release(r)
    assert engine.runner.graph_replays >= 3 and int(engine.runner.status) == 0


@pytest.mark.gpu
def test_a_step_above_the_limit_of_bytes_stays_in_the_latent_space(model, calls, monkeypatch):
    from edgerag_b200.parts.latent_attention import LatentAttention

    folder, raw, forward = model("gates_sinks")
    engine = _engine(folder)
    tokens = _tokens(raw, 300, 1)
    # 300 keys are bounded by 320 rows of at most 3 heads of 192 entries: the first portion (128 keys) fits, the others do not
    monkeypatch.setattr(LatentAttention, "WIDE_MAX_BYTES", 2 * 128 * 3 * 192)
    engine.runner.admit(0)
    _close(_feed(engine.runner, 0, tokens, [120, 100, 80]), forward(tokens), "limit")
    assert len(calls) == 3
