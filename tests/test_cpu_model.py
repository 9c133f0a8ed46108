"""CPU tests of the SciAgent decoder: hand-scheduled backward vs autograd, training, checkpoint
round trip with exact resume, cached generation vs full recompute, reference checkpoint."""
import math
import os
import weakref

import pytest
import torch

from scirust_b200.io import checkpoint as CK
from scirust_b200.models import GQADecoder, SciAgentConfig
from scirust_b200.models.infer import InferenceEngine, reference_generate
from scirust_b200.train import Trainer, TrainerConfig, WarmupCosineSchedule

# golden files of the reference implementation: a checkout beside this repository, or SCIRUST_REFERENCE_DIR
REF = os.environ.get("SCIRUST_REFERENCE_DIR") or os.path.normpath(
    os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "..", "reference"))
CFG = SciAgentConfig(256, 64, 2, 4, 2, 128, 128, 10000.0)


def _ref_loss(m, inp, tgt):
    cfg = m.cfg
    B, S = inp.shape
    H, Hkv, dh = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
    P = {n: p.detach().float().requires_grad_(True) for n, p, _ in m.ordered_params()}
    x = P["embed"][inp.reshape(-1)]
    rms = lambda x, w: x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + cfg.eps) * w  # noqa: E731
    ang = torch.arange(S).float()[:, None] * (cfg.rope_theta ** (-2 * torch.arange(dh // 2).float() / dh))[None]
    c, s_ = torch.cos(ang), torch.sin(ang)

    def rope(t, nh):
        t = t.view(B, S, nh, dh // 2, 2)
        x0, x1 = t[..., 0], t[..., 1]
        return torch.stack((x0 * c[None, :, None] - x1 * s_[None, :, None], x0 * s_[None, :, None] + x1 * c[None, :, None]),
                           -1).view(B, S, nh, dh)
    for i in range(cfg.n_layers):
        qkv = rms(x, P[f"layers.{i}.rms_attn"]) @ P[f"layers.{i}.wqkv"]
        q = rope(qkv[:, :H * dh], H).transpose(1, 2)
        k = rope(qkv[:, H * dh:(H + Hkv) * dh], Hkv).transpose(1, 2).repeat_interleave(H // Hkv, 1)
        v = qkv[:, (H + Hkv) * dh:].view(B, S, Hkv, dh).transpose(1, 2).repeat_interleave(H // Hkv, 1)
        sc = (q @ k.transpose(-1, -2) / math.sqrt(dh)).masked_fill(torch.triu(torch.ones(S, S, dtype=torch.bool), 1), float("-inf"))
        x = x + (torch.softmax(sc, -1) @ v).transpose(1, 2).reshape(B * S, H * dh) @ P[f"layers.{i}.wo"]
        gu = rms(x, P[f"layers.{i}.rms_ffn"]) @ P[f"layers.{i}.wgu"]
        x = x + (torch.nn.functional.silu(gu[:, :cfg.d_ff]) * gu[:, cfg.d_ff:]) @ P[f"layers.{i}.wd"]
    logits = rms(x, P["rms_final"]) @ P["embed"].t()
    return torch.nn.functional.cross_entropy(logits, tgt.reshape(-1)), P


def test_block_backward_matches_autograd():
    m = GQADecoder(CFG, seed=1)
    tok = torch.randint(0, 256, (2, 33), generator=torch.Generator().manual_seed(0))
    inp, tgt = tok[:, :-1], tok[:, 1:]
    m.zero_grad_flags()
    loss = m(inp, tgt)
    loss.backward()
    rl, P = _ref_loss(m, inp, tgt)
    rl.backward()
    assert abs(float(loss) - float(rl)) < 2e-3
    for n, p, _ in m.ordered_params():
        rel = (p.main_grad.float() - P[n].grad).norm() / (P[n].grad.norm() + 1e-12)
        assert rel < 0.02, (n, float(rel))


def test_training_reduces_loss_and_resume_is_exact(tmp_path):
    tok = torch.randint(0, 256, (2, 33), generator=torch.Generator().manual_seed(0))
    m = GQADecoder(CFG, seed=1)
    tr = Trainer(m, TrainerConfig(lr=1e-2, weight_decay=0.0))
    losses = [float(tr.train_step(tok)) for _ in range(6)]
    assert losses[-1] < losses[0]
    CK.save_sciagent_checkpoint(m, tmp_path / "step_6", 6, losses[-1], 1e-2, trainer=tr)
    assert CK.latest_checkpoint(tmp_path).name == "step_6"
    m2, meta = CK.load_sciagent_checkpoint(tmp_path / "step_6")
    assert meta["step"] == 6 and meta["config"].d_ff == CFG.d_ff and meta["config"].eps == pytest.approx(CFG.eps)
    tr2 = Trainer(m2, TrainerConfig(lr=1e-2, weight_decay=0.0))
    CK.load_optimizer_state(m2, tr2, tmp_path / "step_6")
    assert float(tr.train_step(tok)) == float(tr2.train_step(tok)) and torch.equal(m.flat, m2.flat)
    # non-finite gradients skip the update
    before = m.flat.clone()
    bad = Trainer(m, TrainerConfig(lr=1e-2))
    bad.master.copy_(m.flat.float())
    m.embed.data[0, 0] = float("nan")
    bad.master[0] = float("nan")
    bad.train_step(tok)
    assert torch.equal(m.flat[8:], before[8:])
    (tmp_path / "step_10").mkdir()
    (tmp_path / "step_900").mkdir()
    assert CK.latest_checkpoint(tmp_path) is None or CK.latest_checkpoint(tmp_path).name != "step_6"
    CK.prune_checkpoints(tmp_path, 1)
    assert [d.name for d in tmp_path.iterdir() if d.name.startswith("step_")] == ["step_900"]


def test_reference_state_dict_roundtrip_and_names():
    m = GQADecoder(CFG, seed=2)
    sd = m.reference_state_dict()
    assert "sciagent.layer0.attn.wk.weight" in sd and "sciagent.layer1.rms_ffn/weight" in sd
    assert tuple(sd["sciagent.layer0.attn.wk.weight"].shape) == (64, 32) and tuple(sd["sciagent.rms_final/weight"].shape) == (1, 64)
    m2 = GQADecoder(CFG, seed=3)
    m2.load_reference_state_dict(sd)
    assert torch.equal(m.flat, m2.flat)
    del sd["sciagent.layer0.ffn.up.weight"]
    with pytest.raises(KeyError):
        m2.load_reference_state_dict(sd)


def test_cached_paged_generation_equals_full_recompute():
    m = GQADecoder(CFG, seed=1, init_std=0.2)
    p = torch.randint(1, 256, (2, 9), generator=torch.Generator().manual_seed(0))
    eng = InferenceEngine(m, max_batch=2, max_seq=64, page=8)
    a = eng.generate(p, 6)
    assert torch.equal(a, reference_generate(m, p, 6))
    assert torch.equal(a, eng.generate(p, 6))       # engine is reusable
    q8 = InferenceEngine(m, quant="int8", max_batch=2, max_seq=64, page=8).generate(p, 6)
    assert (q8 == a).float().mean() > 0.5
    with pytest.raises(ValueError):
        eng.generate(p, 100)


def test_engine_with_a_product_of_its_own():
    """A subclass whose ``_linear`` takes the activations, the matrix and a residual, and nothing else."""
    class Adapted(InferenceEngine):
        def _linear(self, x, w, residual=None):
            return InferenceEngine._linear(self, x, w, residual)

    m = GQADecoder(CFG, seed=1, init_std=0.2)
    p = torch.randint(1, 256, (10, 9), generator=torch.Generator().manual_seed(0))
    a, b = (cls(m, max_batch=10, max_seq=32, page=8).generate(p, 4) for cls in (Adapted, InferenceEngine))
    assert torch.equal(a, b)


def test_memory_that_runs_out_beside_matrices_expanded_ahead():
    """A piece of a layer is run again with those matrices given back, and with nothing left of what the first run had allocated;
    where none had been expanded the error is the caller's."""
    from scirust_b200.models.infer import _WidenAhead

    class Block:
        pass

    alive = []

    def part(runs):
        mine = Block()
        alive.append(weakref.ref(mine))
        if len(alive) <= runs:
            raise torch.OutOfMemoryError("no memory")
        assert alive[0]() is None
        return 7

    def plan(taken):
        alive.clear()
        p = _WidenAhead([], 0)
        p.order, p.wide, p.taken = ["a", "b"], {1: early} if taken else {}, taken
        return p

    early = Block()
    p = plan(1)
    gone = weakref.ref(early)
    del early
    assert p.run(part, 1) == 7 and p.ran_out and len(alive) == 2 and gone() is None
    assert p.product("c") == ("c", {})
    with pytest.raises(torch.OutOfMemoryError):       # once per plan
        p.run(lambda: part(99))
    early = Block()
    for taken in (1, 0):                              # both runs fail; nothing was expanded ahead
        p = plan(taken)
        with pytest.raises(torch.OutOfMemoryError):
            p.run(part, 99)
        assert len(alive) == 1 + taken and p.ran_out is bool(taken)


def test_warmup_cosine_schedule():
    s = WarmupCosineSchedule(1.0, 0.1, 10, 110)
    assert s.lr_at(0) == 0.0 and s.lr_at(5) == pytest.approx(0.5) and s.lr_at(10) == pytest.approx(1.0)
    assert s.lr_at(60) == pytest.approx(0.55, abs=1e-6) and s.lr_at(500) == pytest.approx(0.1)


@pytest.mark.skipif(not os.path.isfile(f"{REF}/scirust-sciagent/checkpoints/small-20M/final/model.safetensors"),
                    reason="reference tree not mounted")
def test_shipped_reference_checkpoint_predicts_source_text():
    from scirust_b200.tokenizer import BpeTokenizer
    m, meta = CK.load_sciagent_checkpoint(f"{REF}/scirust-sciagent/checkpoints/small-20M/final")
    assert meta["step"] == 2000 and m.num_params() == 1639552
    tok = BpeTokenizer.load_json(f"{REF}/scirust-sciagent/tokenizer/bpe.json")
    ids = tok.encode(open(f"{REF}/scirust-core/src/nn/linear.rs").read()[:6000])[:257]
    t = torch.tensor([ids])
    with torch.no_grad():
        loss = float(m(t[:, :-1], t[:, 1:]))
    assert loss < 7.0          # ln(8192) = 9.01 for a model that knows nothing


def test_library_baseline_model_computes_the_same_loss():
    """The stock-PyTorch arm of the benchmark is the same network: with the native model's weights its
    loss agrees to bf16 accuracy."""
    from scirust_b200.models.baseline_torch import TorchLibraryDecoder
    cfg = SciAgentConfig(vocab_size=128, d_model=64, n_layers=2, n_heads=4, n_kv_heads=2, d_ff=128, max_seq_len=32)
    ours = GQADecoder(cfg, device="cpu", seed=5, init_std=0.05)
    lib = TorchLibraryDecoder(cfg, device="cpu", seed=0)
    with torch.no_grad():
        lib.embed.copy_(ours.embed)
        lib.rms_final.copy_(ours.rms_final)
        for a, b in zip(lib.blocks, ours.layers):
            for n in ("rms_attn", "rms_ffn", "wqkv", "wo", "wgu", "wd"):
                getattr(a, n).copy_(getattr(b, n))
    toks = torch.randint(0, 128, (2, 17), generator=torch.Generator().manual_seed(3))
    l_ours = ours(toks[:, :-1], toks[:, 1:]).float().item()
    l_lib = lib(toks[:, :-1], toks[:, 1:]).float().item()
    assert abs(l_ours - l_lib) < 3e-2, (l_ours, l_lib)


def test_corpus_filter_dedup_split_and_muon_train_optimizer(tmp_path):
    import numpy as np
    from scirust_b200.autodiff import Tape, TrainOptimizer
    from scirust_b200.data import corpus as CP
    from scirust_b200.train.schedule import WarmupCosineSchedule

    assert CP.parse_extensions(".rs, PY,,md") == ["rs", "py", "md"]
    assert CP.skip_source_dir("node_modules") and not CP.skip_source_dir("src")
    assert CP.content_hash("") == 0xCBF29CE484222325 and CP.content_hash("a") == 0xAF63DC4C8601EC8C
    assert CP.source_quality("x.rs", "   \n") == "empty"
    assert CP.source_quality("Cargo.lock", "[[package]]") is not None
    assert CP.source_quality("a.rs", "// @generated by tool\nfn main() {}\n") == "declared generated"
    assert CP.source_quality("a.js", "x" * 12000) == "minified (giant line)"
    assert CP.source_quality("t.csv", ("1234567890," * 30 + "\n") * 3) is not None
    good = "//! module\nuse std::collections::HashMap;\nfn add(a: i32, b: i32) -> i32 { a + b }\n" * 5
    assert CP.source_quality("lib.rs", good) is None

    tr, va = CP.distributed_window_split(100_001, 100, 0.1)
    assert len(tr) + len(va) == 1000 and not set(tr) & set(va) and 60 <= len(va) <= 140
    assert (tr, va) == CP.distributed_window_split(100_001, 100, 0.1)
    assert CP.distributed_window_split(50, 100, 0.1) == ([], [])
    t2, v2 = CP.distributed_window_split(201, 100, 0.1)
    assert len(t2) == 1 and len(v2) == 1

    src = tmp_path / "src"
    (src / "node_modules").mkdir(parents=True)
    (src / "a.rs").write_text(good)
    (src / "b.rs").write_text(good)                    # exact duplicate
    (src / "c.rs").write_text("// do not edit\n" + good)
    (src / "node_modules" / "d.rs").write_text(good + "// other\n")
    (src / "e.txt").write_text(good)

    class ByteTok:
        def encode(self, text):
            return list(text.encode())
    rep = CP.collect_corpus(src, ["rs"], ByteTok(), tmp_path / "shard.bin")
    assert rep["files_kept"] == 1 and rep["duplicates"] == 1 and rep["dropped"] == {"declared generated": 1}
    ld = CP.ShardLoader()
    ld.load_dir(tmp_path)
    assert ld.total_tokens() == rep["tokens"] == len(good.encode()) + 1
    assert CP.token_stream_hash(ld.tokens()) == rep["token_stream_hash"]
    ds = CP.PretrainDataset(np.array([0, 1, 2, 200, 4, 5, 6, 7, 8]), 4, 10)
    x, y = ds.next_batch(1)
    assert x == [0, 1, 2, 3] and y == [1, 2, 3, 4]      # 200 is out of vocabulary -> <unk> = 3
    a, b = CP.PretrainDataset(np.arange(60), 5, 100), CP.PretrainDataset(np.arange(60), 5, 100)
    a.shuffle(42)
    b.shuffle(42)
    assert a.next_batch(2) == b.next_batch(2) and a.starts != sorted(a.starts)

    # Muon / Adam behind TrainOptimizer drive a tape regression downhill; the schedule sets the rate
    torch.manual_seed(0)
    X, Wt = torch.randn(32, 6), torch.randn(6, 3)
    Y = X @ Wt
    for make in (TrainOptimizer.new_muon, TrainOptimizer.new_adam):
        W0 = torch.zeros(6, 3)
        opt = make(0.05).with_weight_decay(0.0)
        sched = WarmupCosineSchedule(0.05, 0.005, 5, 120)
        first = last = None
        for step in range(120):
            tape = Tape()
            w = tape.input(W0)
            diff = tape.constant(X).matmul(w).sub(tape.constant(Y))
            loss = diff.mul(diff).sum()
            tape.backward(loss)
            opt.apply_schedule(sched, step)
            opt.step([w.idx], tape)
            W0 = tape.value(w.idx).t.clone()
            first = first if first is not None else loss.item()
            last = loss.item()
        assert last < 0.2 * first, (make.__name__, first, last)
        assert abs(opt.lr - sched.lr_at(119)) < 1e-9


def test_activation_recompute_gives_identical_gradients_and_losses():
    """Backward that re-runs each block's forward from the saved block input produces the bits of the backward that
    kept every activation (same kernels, same reduction orders), step after step."""
    from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
    from scirust_b200.train.trainer import Trainer, TrainerConfig
    cfg = SciAgentConfig(vocab_size=96, d_model=32, n_layers=3, n_heads=4, n_kv_heads=2, d_ff=64, max_seq_len=32)
    g = torch.Generator().manual_seed(0)
    toks = torch.randint(0, cfg.vocab_size, (4, 3, 17), generator=g)
    losses, flats = [], []
    for rec in (False, True):
        m = GQADecoder(cfg, device=torch.device("cpu"), seed=5)
        tr = Trainer(m, TrainerConfig(lr=1e-2, activation_recompute=rec))
        assert m.activation_recompute == rec
        losses.append([float(tr.train_step(t)) for t in toks])
        flats.append(m.flat.clone())
    assert losses[0] == losses[1]
    assert torch.equal(flats[0], flats[1])
