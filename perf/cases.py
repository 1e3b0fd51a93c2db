"""The work that users have this library do, as cases that can be timed and compared.

A case is one pass through the public entry points over an LFM3 model with weights made from a seed:

  logits   one prompt through `Model.logits` (scoring, first token)
  append   a saved conversation is resumed and gets `new` more tokens at once (`Model.resume_checkpoint`,
           `Session.append_logits`)
  portions a long prompt that comes in portions of `portion` tokens (`Engine.step` with nothing wanted but at the end)
  resume   `batch` sequences go on from saved conversations by `steps` given tokens each, one `Engine.step` per token: decode
  wave     `batch` prompts of unequal lengths start in one step, then get `steps` given tokens each

The tokens are given (a replay), so that every pass computes the same and logits can be compared; the recorded decode step
chooses the next token on the device all the same.  The model sizes are those of `bench.py`'s three configurations and of the
tests' tiny configuration.
"""
import math

import torch

from catena_models_b200 import Model
from catena_models_b200.engine.model import DecoderModel


def _attention_every_third(layers):
    return ["conv" if l % 3 != 2 else "full_attention" if l % 6 == 2 else "sliding_attention" for l in range(layers)]


def _attention_at(layers, at, alternate):
    kinds = {l: "sliding_attention" if alternate and i % 2 else "full_attention" for i, l in enumerate(at)}
    return [kinds.get(l, "conv") for l in range(layers)]


# name: hidden, feed-forward, heads, key/value heads, head size, vocabulary, window, rotation base, kinds of layers
MODELS = {
    "tiny": (64, 176, 4, 2, 16, 256, 16, 10000.0, ["conv", "sliding_attention", "conv", "full_attention"]),
    "350m": (1024, 4608, 16, 8, 64, 65536, 4096, 1000000.0, _attention_at(16, (2, 5, 8, 10, 12, 14), False)),
    "1.7b": (2048, 8192, 32, 8, 64, 65536, 4096, 1000000.0, _attention_every_third(24)),
    "2.6b": (2048, 10752, 32, 8, 64, 65536, 4096, 1000000.0, _attention_at(30, (2, 6, 10, 14, 18, 22, 26, 29), True)),
}
CONTEXT = 32768
TAPS = 3
EPS = 1e-5


def _config(name):
    hidden, ffn, heads, kv, hd, vocab, window, theta, kinds = MODELS[name]
    return dict(architecture="lfm3", vocab_size=vocab, hidden_size=hidden, intermediate_size=ffn, num_hidden_layers=len(kinds),
                layer_types=kinds, num_attention_heads=heads, num_key_value_heads=kv, head_dim=hd, conv_L_cache=TAPS,
                sliding_window=window, rope_theta=theta, norm_eps=EPS, tie_word_embeddings=True, max_position_embeddings=CONTEXT)


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest calls, where launches and the host count: the 32-bit engine on a tiny model, three prompts of a few
        # tokens started together and a few steps on top
        dict(name="tiny f32 wave of 3", kind="wave", model="tiny", dtype="float32", batch=3, shortest=5, longest=17, steps=8),
        # the first token of a short question
        dict(name="1.7b prompt of 77", kind="logits", model="1.7b", dtype="bfloat16", tokens=77),
        # a prompt of ordinary length
        dict(name="1.7b prompt of 2048", kind="logits", model="1.7b", dtype="bfloat16", tokens=2048),
        # the next turn of a chat: a few hundred tokens on top of what the conversation holds
        dict(name="1.7b append 333 on 1900", kind="append", model="1.7b", dtype="bfloat16", held=1900, new=333),
        # one conversation being answered
        dict(name="1.7b decode b1", kind="resume", model="1.7b", dtype="bfloat16", batch=1, shortest=2048, longest=2048, steps=32),
        # a small batch, the benchmark's headline
        dict(name="1.7b decode b8", kind="resume", model="1.7b", dtype="bfloat16", batch=8, shortest=2048, longest=2048, steps=32),
        # a full batch at unequal lengths towards the end of a 4,096-token context
        dict(name="1.7b decode b64", kind="resume", model="1.7b", dtype="bfloat16", batch=64, shortest=1500, longest=4000, steps=32),
        # many unequal prompts started together on a small model, and the tokens that follow
        dict(name="350m wave of 64", kind="wave", model="350m", dtype="bfloat16", batch=64, shortest=16, longest=2048, steps=32),
        # a document as one prompt
        dict(name="2.6b prompt of 16384", kind="logits", model="2.6b", dtype="bfloat16", tokens=16384),
        # the same kind of prompt as a server hands it over, in blocks of 1,024
        dict(name="2.6b prompt in portions", kind="portions", model="2.6b", dtype="bfloat16", tokens=9001, portion=1024),
        # answers over long documents
        dict(name="2.6b decode b20 long", kind="resume", model="2.6b", dtype="bfloat16", batch=20, shortest=9000, longest=16000, steps=32),
        # the 32-bit engine at a real size: prompts and a few tokens, as the checks of a replay run it
        dict(name="350m f32 wave of 4", kind="wave", model="350m", dtype="float32", batch=4, shortest=100, longest=400, steps=8),
    ]


def _cost(case):
    w = work(case)
    return w["bytes"] / 6e12 + w["flops"] / (1.2e15 if case["dtype"] == "bfloat16" else 4e13)


def draw(rng):
    """One more case: the kind by use, sizes over their whole range (over the logarithm where it spans more than a factor of ten)."""
    def log_between(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["resume", "resume", "resume", "logits", "logits", "wave", "append", "portions"])
        dtype = "float32" if rng.random() < 0.1 else "bfloat16"
        model = rng.choice(["350m", "1.7b", "2.6b"])
        if dtype == "float32":
            model, kind = rng.choice(["tiny", "350m"]), "wave"
        case = dict(kind=kind, model=model, dtype=dtype)
        if kind == "logits":
            case.update(tokens=log_between(8, 16384))
        elif kind == "append":
            case.update(held=log_between(64, 12000), new=log_between(2, 2000))
        elif kind == "portions":
            case.update(tokens=log_between(2000, 12000), portion=rng.choice([256, 512, 1000, 1024, 2048]))
        elif kind == "resume":
            longest = log_between(64, 16000)
            case.update(batch=log_between(1, 64), shortest=rng.randint(max(32, longest // 3), longest), longest=longest, steps=rng.randint(12, 40))
        else:
            longest = log_between(16, 2048) if dtype == "bfloat16" else log_between(16, 400)
            case.update(batch=log_between(2, 64) if dtype == "bfloat16" else rng.randint(2, 6), shortest=rng.randint(5, min(64, longest)),
                        longest=longest, steps=rng.randint(4, 40) if dtype == "bfloat16" else rng.randint(2, 8))
        if _cost(case) <= most and _held(case) <= 200000:
            return case


# ------------------------------------------------------------------------------------------------ inputs
SAVED = 4                                  # distinct saved conversations of a "resume" case (sequence b goes on from number b % SAVED)


def _lengths(case, count):
    """`count` lengths from shortest to longest, evenly, in a fixed order that is not sorted."""
    lo, hi = case["shortest"], case["longest"]
    lengths = [lo + (hi - lo) * i // max(1, count - 1) for i in range(count)]
    stride = next(s for s in range(max(1, int(count * 0.618)), 2 * count + 2) if math.gcd(s, count) == 1)
    return [lengths[(i * stride) % count] for i in range(count)]


def _plan(case):
    """(lengths of the prompts that start together, lengths saved beforehand, tokens given per sequence afterwards)."""
    kind = case["kind"]
    if kind in ("logits", "portions"):
        return [case["tokens"]], [], 0
    if kind == "append":
        return [], [case["held"]], case["new"]
    if kind == "resume":
        return [], _lengths(case, min(SAVED, case["batch"])), case["steps"]
    return _lengths(case, case["batch"]), [], case["steps"]


def _held(case):
    """Tokens that the cache holds at most, each sequence rounded up to pages of 64 with one to spare."""
    starts, saved, more = _plan(case)
    up = lambda n: (n + 63) // 64 * 64 + 64  # noqa: E731
    total = sum(up(n + more) for n in starts) + sum(up(n) for n in saved)
    if saved:
        total += sum(up(saved[b % len(saved)] + more) for b in range(case.get("batch", 1)))
    return total


def _weights(case, seed):
    """{name: tensor} on the device, in the types a checkpoint stores: matrices N(0, 0.02), norms around one, what a sublayer adds
    small beside the stream, as trained models have it."""
    hidden, ffn, heads, kv, hd, vocab, _, _, kinds = MODELS[case["model"]]
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    out = {}

    def normal(name, *shape, mean=0.0, std=0.02, dtype=torch.bfloat16):
        out[name] = torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=g)

    f32 = torch.float32
    normal("model.embed_tokens.weight", vocab, hidden, std=0.05)
    normal("model.norm.weight", hidden, mean=1.0, std=0.1, dtype=f32)
    out["rope_freqs.weight"] = torch.empty(hd // 2, dtype=f32, device="cuda").uniform_(1.0, 4.0, generator=g)
    for l, k in enumerate(kinds):
        p = "model.layers.%d." % l
        for n, mean in (("attn_norm", 1.0), ("ffn_norm", 1.0), ("post_attention_norm", 0.006), ("post_ffw_norm", 0.006)):
            normal(p + n + ".weight", hidden, mean=mean, std=0.1 * mean, dtype=f32)
        if k == "conv":
            normal(p + "shortconv.in_proj.weight", 3 * hidden, hidden)
            normal(p + "shortconv.conv.weight", hidden, TAPS, std=0.3, dtype=f32)
            normal(p + "shortconv.out_proj.weight", hidden, hidden)
        else:
            normal(p + "attn_q.weight", heads * hd, hidden)
            normal(p + "attn_k.weight", kv * hd, hidden)
            normal(p + "attn_v.weight", kv * hd, hidden)
            normal(p + "attn_gate.weight", heads, hidden)
            normal(p + "attn_q_norm.weight", hd, mean=1.0, std=0.1, dtype=f32)
            normal(p + "attn_k_norm.weight", hd, mean=1.0, std=0.1, dtype=f32)
            normal(p + "attn_output.weight", hidden, heads * hd)
        normal(p + "ffn_gate.weight", ffn, hidden)
        normal(p + "ffn_up.weight", ffn, hidden)
        normal(p + "ffn_down.weight", hidden, ffn)
    return out


def _tokens(case, seed):
    """(prompts that start together, prompts saved beforehand, given tokens [sequence][step]) as lists of ids."""
    vocab = MODELS[case["model"]][5]
    g = torch.Generator().manual_seed(7919 * seed + 5)
    ids = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()  # noqa: E731
    starts, saved, more = _plan(case)
    return [ids(n) for n in starts], [ids(n) for n in saved], [ids(more) for _ in range(case.get("batch", 1))]


# ------------------------------------------------------------------------------------------------ the library's side
class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    s.starts, saved, s.given = _tokens(case, seed)
    config = _config(case["model"])
    decoder = DecoderModel.from_tensors(config, _weights(case, seed), torch.float32 if case["dtype"] == "float32" else torch.bfloat16)
    batch = case.get("batch", 1)
    s.model = Model(decoder, max_tokens=_held(case), max_seqs=batch + len(saved) + 1)
    s.saved = []
    for prompt in saved:
        session = s.model.session(CONTEXT)
        s.model.engine.step([session.slot], [prompt], [[]])
        s.saved.append(session.into_checkpoint())
    steps = case.get("steps", 0)
    s.by_step = [[[row[i]] for row in s.given] for i in range(steps)]
    s.logits = torch.empty((steps, batch, config["vocab_size"]), dtype=torch.float32, device="cuda") if steps else None
    return s


def _given_steps(s, slots):
    engine = s.model.engine
    for i, tokens in enumerate(s.by_step):
        s.logits[i].copy_(engine.step(slots, tokens))


def run(s):
    case, model, engine = s.case, s.model, s.model.engine
    kind = case["kind"]
    if kind == "logits":
        return model.logits(s.starts[0])
    if kind == "append":
        with model.resume_checkpoint(s.saved[0]) as session:
            return session.append_logits(s.given[0])
    if kind == "portions":
        prompt, n = s.starts[0], case["portion"]
        with model.session(len(prompt)) as session:
            for at in range(0, len(prompt), n):
                logits = engine.step([session.slot], [prompt[at:at + n]], None if at + n >= len(prompt) else [[]])
            return logits
    if kind == "resume":
        sessions = [model.resume_checkpoint(s.saved[b % len(s.saved)]) for b in range(case["batch"])]
        _given_steps(s, [x.slot for x in sessions])
        for x in sessions:
            x.close()
        return s.logits
    slots = engine.admit(case["batch"])
    first = engine.step(slots, s.starts)
    _given_steps(s, slots)
    engine.release(slots)
    return first, s.logits


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    hidden, ffn, heads, kv, hd, vocab, window, _, kinds = MODELS[case["model"]]
    size = 4 if case["dtype"] == "float32" else 2
    conv, attn = kinds.count("conv"), len(kinds) - kinds.count("conv")
    matrices = conv * 4 * hidden * hidden + attn * (hidden * hd * 2 * (heads + kv) + heads * hidden) + len(kinds) * 3 * hidden * ffn
    matrix_bytes = 2 * (matrices + vocab * hidden)          # stored in bfloat16; the 32-bit engine keeps them widened
    if case["dtype"] == "float32":
        matrix_bytes *= 2
    kv_row = 2 * kv * hd * size
    total = {"bytes": 0.0, "flops": 0.0}

    def step(past, new, wanted):
        """One step: sequences that hold `past` tokens get `new` each; logits at `wanted` places."""
        rows = sum(new)
        seen = reads = 0
        for k in kinds:
            if k == "conv":
                continue
            w = window if k == "sliding_attention" else 0
            for p, n in zip(past, new):
                whole = n * p + n * (n + 1) / 2             # pairs of a query and a key at or before it
                if w and p + n > w:                         # less those that have left the window
                    out = p + n - w
                    whole -= out * (out + 1) / 2 - (out - n) * (out - n + 1) / 2 if out > n else out * (out + 1) / 2
                seen += whole
                reads += min(p, w) if w else p
        total["bytes"] += matrix_bytes + rows * hidden * size + (reads + attn * rows) * kv_row
        total["bytes"] += conv * len(new) * 2 * (TAPS - 1) * hidden * 4 + wanted * vocab * 4
        total["flops"] += 2.0 * matrices * rows + 4.0 * heads * hd * seen + 2.0 * vocab * hidden * wanted

    starts, saved, more = _plan(case)
    if case["kind"] == "portions":
        n, all_ = case["portion"], case["tokens"]
        for at in range(0, all_, n):
            step([at], [min(n, all_ - at)], 1 if at + n >= all_ else 0)
    elif case["kind"] == "append":
        step(saved, [more], 1)
    else:
        past = list(starts) or [saved[b % len(saved)] for b in range(case["batch"])]
        if starts:
            step([0] * len(starts), starts, len(starts))
        for i in range(more):
            step([p + i for p in past], [1] * len(past), len(past))
    return total


def tolerance(case):
    # Two implementations at these precisions differ in the order of their sums.  bfloat16: activations are rounded after every
    # product, so a sum that falls on the other side of a rounding border shifts what follows by 2^-8 of a value.
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.03, "max": 0.5}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
class _Plain:
    """The decoder in float64, whole sequences of one length at a time on top of a common past."""

    def __init__(self, case, seed):
        self.config = _config(case["model"])
        self.w = {k: v.double() for k, v in _weights(case, seed).items()}

    @staticmethod
    def _norm(x, w):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w

    def _rotate(self, u, first, sliding):
        """u [b, n, heads, hd] at positions first.. ; the angle is a 32-bit product of position and rate, as the model defines it."""
        hd = u.shape[-1]
        rate = torch.tensor([self.config["rope_theta"]], dtype=torch.float32) ** (
            -torch.arange(0, hd, 2, dtype=torch.float32) / hd)
        rate = rate.cuda()
        if not sliding:
            rate = rate / self.w["rope_freqs.weight"].float()
        angle = (torch.arange(first, first + u.shape[1], dtype=torch.float32, device="cuda")[:, None] * rate[None]).double()
        cos, sin = angle.cos()[None, :, None], angle.sin()[None, :, None]
        lo, hi = u[..., :hd // 2], u[..., hd // 2:]
        return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], -1)

    def _attention(self, n, p, sliding, past):
        c, w = self.config, self.w
        b, t, _ = n.shape
        heads, kv, hd = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
        first = past[0].shape[0] if past else 0
        q = self._rotate(self._norm((n @ w[p + "attn_q.weight"].T).view(b, t, heads, hd), w[p + "attn_q_norm.weight"]), first, sliding)
        k = self._rotate(self._norm((n @ w[p + "attn_k.weight"].T).view(b, t, kv, hd), w[p + "attn_k_norm.weight"]), first, sliding)
        v = (n @ w[p + "attn_v.weight"].T).view(b, t, kv, hd)
        out = torch.empty_like(q)
        reach = c["sliding_window"] if sliding else 0
        for i in range(b):
            ks, vs = (torch.cat([past[0], k[i]]), torch.cat([past[1], v[i]])) if past else (k[i], v[i])
            for at in range(0, t, 512):
                to = min(t, at + 512)
                lo = max(0, first + at - reach + 1) if reach else 0
                keys = torch.arange(lo, first + to, device="cuda")
                pos = torch.arange(first + at, first + to, device="cuda")[:, None]
                hidden = keys[None] > pos
                if reach:
                    hidden |= keys[None] + reach <= pos
                qg = q[i, at:to].view(to - at, kv, heads // kv, hd)
                s = torch.einsum("tkgd,skd->kgts", qg, ks[lo:first + to]) * hd ** -0.5
                s = s.masked_fill_(hidden, float("-inf")).softmax(-1)
                out[i, at:to] = torch.einsum("kgts,skd->tkgd", s, vs[lo:first + to]).reshape(to - at, heads, hd)
        out = out * torch.sigmoid(n @ w[p + "attn_gate.weight"].T)[..., None]
        return out.reshape(b, t, heads * hd) @ w[p + "attn_output.weight"].T, (k, v)

    def _conv(self, n, p, past):
        w, hidden = self.w, n.shape[-1]
        gate_in, gate_out, x = (n @ w[p + "shortconv.in_proj.weight"].T).split(hidden, -1)
        bx = gate_in * x
        before = past.expand(n.shape[0], -1, -1) if past is not None else torch.zeros(n.shape[0], TAPS - 1, hidden, dtype=n.dtype, device="cuda")
        s = torch.cat([before, bx], 1)
        z = sum(w[p + "shortconv.conv.weight"][:, j] * s[:, j:j + n.shape[1]] for j in range(TAPS))
        return (z * gate_out) @ w[p + "shortconv.out_proj.weight"].T, s[:, -(TAPS - 1):]

    def __call__(self, rows, past=None, wanted=None):
        """Rows of ids, all of one length, each on top of `past` (what a call with one row gave back).  Logits [rows, wanted
        places, vocabulary] (None: every place) and what one row leaves behind."""
        w = self.w
        h = w["model.embed_tokens.weight"][torch.tensor(rows, device="cuda")]
        left = []
        for l, kind in enumerate(self.config["layer_types"]):
            p = "model.layers.%d." % l
            n = self._norm(h, w[p + "attn_norm.weight"])
            before = past[l] if past else None
            if kind == "conv":
                m, after = self._conv(n, p, before)
                left.append(after[0])
            else:
                m, after = self._attention(n, p, kind == "sliding_attention", before)
                left.append((after[0][0], after[1][0]))
            h = h + self._norm(m, w[p + "post_attention_norm.weight"])
            n = self._norm(h, w[p + "ffn_norm.weight"])
            for i in range(n.shape[0]):                     # a sequence at a time: the feed-forward's rows are wide
                g = n[i] @ w[p + "ffn_gate.weight"].T
                a = g * torch.sigmoid(g) * (n[i] @ w[p + "ffn_up.weight"].T)
                h[i] += self._norm(a @ w[p + "ffn_down.weight"].T, w[p + "post_ffw_norm.weight"])
        n = self._norm(h if wanted is None else h[:, wanted], w["model.norm.weight"])
        return n @ w["model.embed_tokens.weight"].T, left


def exact(case, seed):
    starts, saved, given = _tokens(case, seed)
    plain = _Plain(case, seed)
    if case["kind"] in ("logits", "portions"):
        logits, _ = plain([starts[0]], wanted=[-1])
        return logits[0, 0].cpu() if case["kind"] == "logits" else logits[0]
    if case["kind"] == "append":
        logits, _ = plain([saved[0] + given[0]], wanted=[-1])
        return logits[0, 0].cpu()
    steps, batch, vocab = case["steps"], case["batch"], MODELS[case["model"]][5]
    out = torch.empty((steps, batch, vocab), dtype=torch.float64, device="cuda")
    if case["kind"] == "resume":
        for i, prompt in enumerate(saved):
            _, past = plain([prompt], wanted=[-1])
            for b in range(i, batch, len(saved)):
                out[:, b] = plain([given[b]], past)[0][0]
        return out
    first = torch.empty((batch, vocab), dtype=torch.float64, device="cuda")
    for b, prompt in enumerate(starts):
        logits, _ = plain([prompt + given[b]], wanted=list(range(len(prompt) - 1, len(prompt) + steps)))
        first[b], out[:, b] = logits[0, 0], logits[0, 1:]
    return first, out
