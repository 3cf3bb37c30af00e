"""Workloads of the scoring service, from the smallest request to the longest prefix, through the calls a user makes.

A request is a prefix tree of candidate prompts: a shared root, one stem per question, one tail per candidate. The layers
have the full width of the 27B backbone (modelgen.FULL: hidden 5120, MLP 17408, 24 / 4 attention heads of 256, Gated DeltaNet
with 16 key and 32 value heads of 128); the depth is two periods of the layer pattern, i.e. 8 of the 64 layers (six Gated
DeltaNet, two attention). Every layer of a kind does the same work, so a whole forward is eight times the layers here plus
the same fixed part; the depth is cut because random weights amplify every bf16 rounding from layer to layer, and because
three weight sets (bf16, e4m3, 48 value heads) have to fit one GPU beside each other. 5.7 GB of weights pass per forward, so
nothing of a layer is still in the L2 when it comes round again.

Routes ("route" of a case):
  score    Scorer.score_tokens: token lists in, scores out; the graph of the shape is captured, as in a service whose shapes
           come back
  first    the same call on a scorer that meets each shape for the first time and runs it without a graph
           (capture_after), as for the mixed streams in which hardly a shape repeats
  packed   Scorer.score_packed: several requests in one forward
  state    Scorer.score_state: one question over a long shared context
  hidden   gtree_build + forward_gtree, the final hidden state of every candidate
  batch    FastQwen35.forward: a right-padded batch of independent sequences, every hidden state
A scorer and its weights live as long as the process, as in a service; requests are made from the seed.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "open-jev-fast_b200"))
from ojb200 import fastmodel as FM, modelgen as MG, server as SV, trees  # noqa: E402

LAYERS = 8
VOCAB = MG.FULL["vocab_size"]
ANSWERS = 16                      # rows of the scoring head: a small answer vocabulary
_services = {}


def listed():
    """shape: seed of the stem and tail lengths, which lie within a factor of about 1.6 around stem and tail."""
    base = dict(route="score", fp8=False, heads=32, requests=1, questions=3, candidates=7, shape=1)
    case = lambda name, **over: dict(base, name=name, **over)
    return [
        # a yes/no check on a short message: 30-odd rows, bound by the weights and by the length of the launch chain
        case("score_smallest", root=14, stem=8, tail=3, questions=1, candidates=2),
        # the shape of the example request the service ships with: 280 rows, every candidate with a long tail of its own
        case("score_example", root=30, stem=21, tail=26),
        # the benchmark's request: 540 rows, most of them shared context
        case("score_request", root=420, stem=25, tail=6),
        # a wide request with odd sizes on the checkpoint variant with 48 value heads
        case("score_wide_48_heads", root=651, stem=37, tail=23, candidates=12, heads=48, shape=2),
        # the median and the longest prefix of the service's length sweep
        case("score_prefix_2500", root=2470, stem=22, tail=19, questions=2, candidates=6, shape=3),
        case("score_prefix_16k", root=16384, stem=30, tail=25, candidates=9, shape=4),
        # several waiting requests put into one forward
        case("packed_4_requests", route="packed", requests=4, root=420, stem=25, tail=6),
        # 8-bit projections, for callers that accept their error: the benchmark's request and a long prefix
        case("fp8_request", fp8=True, root=420, stem=25, tail=6),
        case("fp8_prefix_4k", fp8=True, root=4096, stem=24, tail=20, shape=5),
        # one question over a long document, prefix state handed to every candidate
        case("state_document", route="state", root=1900, stem=12, tail=14, questions=1, candidates=5, shape=6),
        # a shape met for the first time: no graph, every launch goes through the host
        case("first_sight", route="first", root=333, stem=17, tail=11, questions=2, candidates=5, shape=7),
        # independent prompts in a padded batch, the plain forward of the backbone
        case("batch_of_6", route="batch", root=180, stem=60, tail=20, questions=6, candidates=6, shape=8),
    ]


def draw(rng):
    route = rng.choice(["score"] * 7 + ["packed", "state", "first", "hidden", "batch"])
    fp8 = route == "score" and rng.random() < 0.2
    heads = 48 if route == "score" and not fp8 and rng.random() < 0.2 else 32
    longest = {"score": 15000, "packed": 1500, "state": 4000, "first": 3000, "hidden": 3000, "batch": 400}[route]
    root = round(math.exp(rng.uniform(math.log(12), math.log(longest))))
    questions = 1 if route == "state" else rng.randint(1, 3)
    candidates = rng.randint(max(2, questions), 12)
    if route == "batch":
        questions = candidates = rng.randint(2, 8)
    return dict(route=route, fp8=fp8, heads=heads, requests=rng.randint(2, 4) if route == "packed" else 1, root=root,
                questions=questions, candidates=candidates, stem=rng.randint(4, 40), tail=rng.randint(2, 40), shape=rng.randrange(1 << 30))


def _lengths(case, index=0):
    """Stem length per question, tail length and question per candidate of one request of the case."""
    r = random.Random(case["shape"] * 31 + index)
    near = lambda n: max(1, round(n * math.exp(r.uniform(-0.5, 0.5))))
    groups = sorted(list(range(case["questions"])) + [r.randrange(case["questions"]) for _ in range(case["candidates"] - case["questions"])])
    return [near(case["stem"]) for _ in range(case["questions"])], [near(case["tail"]) for _ in groups], groups


def _tree(case, seed, index=0):
    stems, tails, groups = _lengths(case, index)
    return trees.make_tree((seed * 64 + index) % (1 << 32), case["root"], stems, tails, groups, VOCAB)


def _service(heads, fp8, first):
    """One model and its scorer, kept for the life of the process."""
    dev = torch.device("cuda", torch.cuda.current_device())
    model = _services.get((heads, fp8))
    if model is None:
        cfg = MG.make_config(**dict(MG.FULL, num_hidden_layers=LAYERS, linear_num_value_heads=heads))
        model = _services[heads, fp8] = FM.FastQwen35(MG.build_core(cfg, device=dev, seed=0), free_original=True, fp8=fp8)
    scorer = _services.get((heads, fp8, first))
    if scorer is None:
        W, b = MG.make_head(model.H, A=ANSWERS, seed=1, device=dev)
        scorer = _services[heads, fp8, first] = SV.Scorer(model, W, b, device=dev, capture_after=(1 << 30) if first else 1)
    return model, scorer


def _batch(case):
    """Lengths of the sequences of a batch: about root + stem + tail tokens, the shortest a third of that."""
    stems, tails, groups = _lengths(case)
    lens = [case["root"] + stems[g] + t for g, t in zip(groups, tails)]
    return [max(1, n * (i + 2) // (len(lens) + 1)) for i, n in enumerate(lens)]


def prepare(case, seed):
    model, scorer = _service(case["heads"], case["fp8"], case["route"] == "first")
    state = dict(route=case["route"], model=model, scorer=scorer)
    if case["route"] == "batch":
        lens = _batch(case)
        dev = model.embed.weight.device
        g = torch.Generator(device=dev).manual_seed(seed)
        state["ids"] = torch.randint(8, VOCAB, (len(lens), max(lens)), generator=g, device=dev)
        state["mask"] = (torch.arange(max(lens), device=dev)[None, :] < torch.tensor(lens, device=dev)[:, None]).long()
        state["ids"] *= state["mask"]
        return state
    make = lambda s: [_tree(case, s, i) for i in range(case["requests"])]
    state["requests"] = make(seed)
    if case["route"] in ("score", "packed", "state"):
        # the service has met the shape before: its graph is captured (once per shape and process) on another request of that shape
        run(dict(state, requests=make(seed + 977)))
    return state


def run(state):
    route, scorer = state["route"], state["scorer"]
    if route == "batch":
        return state["model"].forward(input_ids=state["ids"], attention_mask=state["mask"]).last_hidden_state
    if route == "packed":
        return scorer.score_packed(state["requests"])
    seqs, groups = state["requests"][0]
    if route == "state":
        return scorer.score_state(seqs)
    if route == "hidden":
        ids, lay = state["model"].gtree_build(seqs, groups, 0, dense=False)
        return state["model"].forward_gtree(ids, lay)
    return scorer.score_tokens(seqs, groups)


def work(case):
    """Weights once, token ids in, results out. Products: every row through every layer, but through the last layer's output
    projection and MLP only the rows whose result is asked for."""
    F = MG.FULL
    H, I, D, HQ, HKV = F["hidden_size"], F["intermediate_size"], F["head_dim"], F["num_attention_heads"], F["num_key_value_heads"]
    HK, HV, G = F["linear_num_key_heads"], case["heads"], F["linear_key_head_dim"]
    attn = LAYERS // 4
    lin = LAYERS - attn
    n_lin_in, n_attn_in = 2 * HK * G + 2 * HV * G + 2 * HV, (2 * HQ + 2 * HKV) * D
    lin_w, attn_w = H * n_lin_in + H * HV * G, H * n_attn_in + H * HQ * D
    mlp_w = 3 * H * I
    rows = pairs = results = 0          # distinct token rows, (query, visible key) pairs, rows of the result
    if case["route"] == "batch":
        for n in _batch(case):
            rows, pairs = rows + n, pairs + n * (n + 1) // 2
        results = rows
    else:
        for i in range(case["requests"]):
            stems, tails, groups = _lengths(case, i)
            root = case["root"]
            rows += root + sum(stems) + sum(tails)
            pairs += root * (root + 1) // 2 + sum(n * root + n * (n + 1) // 2 for n in stems)
            pairs += sum(t * (root + stems[g]) + t * (t + 1) // 2 for t, g in zip(tails, groups))
            results += len(tails)
    last = H * HQ * D + mlp_w           # the last layer is an attention layer
    flops = 2.0 * rows * (lin * lin_w + attn * attn_w + LAYERS * mlp_w - last) + 2.0 * results * last
    flops += attn * 4.0 * HQ * D * pairs + lin * 8.0 * rows * HV * G * G
    weights = (lin * lin_w + attn * attn_w + LAYERS * mlp_w) * (1 if case["fp8"] else 2)
    width = H * 2 if case["route"] in ("batch", "hidden") else ANSWERS * 4
    return dict(bytes=float(weights + rows * (H * 2 + 8) + results * width), flops=flops)


def tolerance(case):
    """Runs of the same weights and tokens with other GEMM kernels, other K ranges and the other attention kernel differ by
    rel 6.6e-3 .. 8.1e-3 (max 1.3e-2 .. 3.0e-2) on every bf16 case: eight layers of random weights amplify the bf16 roundings
    of the activations. On e4m3 operands a rounding that falls the other way is a step of 1/8 .. 1/16 of the value: the other
    attention kernel alone moves the results by rel 4.8e-2 (max 0.11)."""
    return {"rel": 0.16, "max": 0.45} if case["fp8"] else {"rel": 2.5e-2, "max": 0.1}
