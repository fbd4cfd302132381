"""The work a user of the decode tail has it do, as cases that can be prepared, run and timed.

Every case goes through the package's public Python calls (each one C-ABI entry point) on buffers such as a serving
loop keeps.  The kinds:

  decode       hidden states -> FP8 head -> top-p sampler: one step of a decode batch (benchmark configurations 2 and 5)
  sample       logits that the model already produced -> token ids, peaked rows as a trained model gives them
               (configuration 1's recipe), with top-p, top-k or greedily
  verify       speculative verification of target rows against draft rows (configuration 3)
  constrained  penalties over the token history, grammar bitmask, top-k and top-p (configuration 4)
  engine       one speculative transaction of one conversation through the engine's own plugin symbols: drafter head,
               Markov bias and draft sampling position by position, final norm, target head, verification
  score        log-normaliser and top-N log-probabilities of a scoring request
  rows         the engine's original row interface: probability rows, then verification on the rows

The vocabulary is the engine's (129280) unless a case says otherwise; hidden sizes are those of the two head formats.
"""
import math

import torch

import __graft_entry__

VOCAB = 129280
FP8_K = 4096      # hidden size of the FP8 head's configurations
PLUGIN_K = 5120   # hidden size of the engine's BF16 / FP32 head plugins
DRAFT_NOISE = 0.30  # draft logits = target + N(0, 0.3^2): about 85 % of the proposals are accepted


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one interactive user: latency and launches
        {"name": "decode_b1", "kind": "decode", "batch": 1, "temperature": 0.6, "top_p": 0.95},
        # a small server
        {"name": "decode_b8", "kind": "decode", "batch": 8, "temperature": 0.6, "top_p": 0.95},
        # the largest batch that is still bound by the weights
        {"name": "decode_b64", "kind": "decode", "batch": 64, "temperature": 0.6, "top_p": 0.95},
        # throughput serving; the head is a large GEMM
        {"name": "decode_b1024", "kind": "decode", "batch": 1024, "temperature": 0.6, "top_p": 0.95},
        # an odd batch over a smaller, odd vocabulary: every second row is unaligned
        {"name": "sample_b19_v50001", "kind": "sample", "rows": 19, "vocab": 50001, "temperature": 0.7, "top_p": 0.95,
         "top_k": 0},
        # one conversation with the longest draft the engine allows
        {"name": "verify_s1_d5", "kind": "verify", "sequences": 1, "drafts": 5, "vocab": VOCAB, "temperature": 0.6,
         "top_p": 0.95},
        # a batch of conversations
        {"name": "verify_s32_d2", "kind": "verify", "sequences": 32, "drafts": 2, "vocab": VOCAB, "temperature": 0.6,
         "top_p": 0.95},
        # a few tool-calling chats with short, unequal histories
        {"name": "constrained_b3", "kind": "constrained", "rows": 3, "history": 1500, "ragged": True, "mask": True,
         "temperature": 0.8, "top_k": 50, "top_p": 0.9},
        # structured output at scale, 32K-token contexts
        {"name": "constrained_b256", "kind": "constrained", "rows": 256, "history": 32768, "ragged": False, "mask": True,
         "temperature": 0.8, "top_k": 50, "top_p": 0.9},
        # the reference engine's own decode loop with two drafts, BF16 heads
        {"name": "engine_d2", "kind": "engine", "drafts": 2, "head": "bf16", "temperature": 0.6, "top_p": 0.95},
        # a score request
        {"name": "score_r5_n20", "kind": "score", "rows": 5, "vocab": VOCAB, "top_n": 20},
        # one transaction of a caller that keeps the row interface
        {"name": "rows_d2", "kind": "rows", "drafts": 2, "vocab": VOCAB, "temperature": 0.7, "top_p": 0.95},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _vocab(rng):
    """Half of the callers run the engine's vocabulary, the others any size up to the library's limit."""
    return VOCAB if rng.random() < 0.5 else _log_int(rng, 16000, 131072)


def draw(rng):
    kind = rng.choices(["decode", "sample", "verify", "constrained", "engine", "score", "rows"],
                       [32, 16, 16, 16, 8, 6, 6])[0]
    t, top_p = round(rng.uniform(0.5, 1.1), 2), rng.choice([0.9, 0.95, 0.99])
    if kind == "decode":
        return {"kind": kind, "batch": _log_int(rng, 1, 1024), "temperature": t, "top_p": top_p}
    if kind == "sample":
        mode = rng.choice(["top_p", "top_p", "top_k", "greedy", "full"])
        return {"kind": kind, "rows": _log_int(rng, 1, 256), "vocab": _vocab(rng),
                "temperature": 0.0 if mode == "greedy" else t, "top_p": 1.0 if mode in ("greedy", "full") else top_p,
                "top_k": rng.randint(5, 64) if mode == "top_k" else 0}
    if kind == "verify":
        return {"kind": kind, "sequences": _log_int(rng, 1, 32), "drafts": rng.randint(1, 5), "vocab": _vocab(rng),
                "temperature": t, "top_p": top_p}
    if kind == "constrained":
        return {"kind": kind, "rows": _log_int(rng, 1, 256), "history": _log_int(rng, 32, 32768),
                "ragged": rng.random() < 0.7, "mask": rng.random() < 0.6, "temperature": t,
                "top_k": rng.choice([0, 20, 50]), "top_p": top_p}
    if kind == "engine":
        return {"kind": kind, "drafts": rng.randint(1, 5), "head": rng.choice(["bf16", "f32"]), "temperature": t,
                "top_p": top_p}
    if kind == "score":
        return {"kind": kind, "rows": _log_int(rng, 1, 64), "vocab": _vocab(rng), "top_n": rng.randint(0, 32)}
    return {"kind": kind, "drafts": rng.randint(1, 5), "vocab": _vocab(rng), "temperature": t, "top_p": top_p}


# ---------------------------------------------------------------------------------------------------------- inputs
class _Inputs:
    """The package, the device and the generator that one prepare() draws everything from."""

    def __init__(self, seed):
        self.pkg = __graft_entry__.load_package()
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, device=self.dev, generator=self.gen)

    def uniform(self, *shape, dtype=torch.float32):
        return torch.rand(*shape, device=self.dev, generator=self.gen, dtype=dtype)

    def empty(self, *shape, dtype):
        return torch.empty(*shape, dtype=dtype, device=self.dev)

    def addresses(self, rows):
        """Philox key and attempt counter of each row (uint64 bit patterns)."""
        return (torch.randint(0, 2 ** 62, (rows,), device=self.dev, generator=self.gen),
                torch.randint(0, 2 ** 20, (rows,), device=self.dev, generator=self.gen))

    def peaked_logits(self, rows, vocab):
        """The benchmark's logits: log-Zipf (s = 1.1) over a permutation of the ids of each row, plus 3 N(0, 1)."""
        zipf = -1.1 * torch.log(torch.arange(1, vocab + 1, device=self.dev, dtype=torch.float32))
        out = 3.0 * self.normal(rows, vocab)
        for r in range(rows):
            out[r, torch.randperm(vocab, device=self.dev, generator=self.gen)] += zipf
        return out

    def fp8_weights(self, n, k):
        """e4m3 weights of N(0, 0.02^2) with one fp32 scale per 128 x 128 block (n and k are multiples of 128)."""
        wq, ws = self.empty(n, k, dtype=torch.uint8), self.empty(n // 128, k // 128, dtype=torch.float32)
        for r0 in range(0, n, 16384):
            r1 = min(n, r0 + 16384)
            blocks = (0.02 * self.normal(r1 - r0, k)).view(-1, 128, k // 128, 128)
            scale = blocks.abs().amax(dim=(1, 3)) / 448.0
            wq[r0:r1] = (blocks / scale[:, None, :, None]).reshape(-1, k).to(torch.float8_e4m3fn).view(torch.uint8)
            ws[r0 // 128:r1 // 128] = scale
        return wq, ws

    def weights(self, n, k, dtype, std):
        w = self.empty(n, k, dtype=dtype)
        for r0 in range(0, n, 16384):
            r1 = min(n, r0 + 16384)
            w[r0:r1] = std * self.normal(r1 - r0, k)
        return w

    def proposals(self, logits, temperature, top_p):
        """One id per row from the top-p nucleus (taken a hair smaller, so that no id lies on its edge)."""
        p, order = torch.softmax(logits.double() / temperature, -1).sort(-1, descending=True)
        mass = p.cumsum(-1)
        keep = mass <= top_p - 1e-6
        keep[:, 0] = True
        kept = (p * keep).cumsum(-1)
        u = self.uniform(logits.shape[0], 1, dtype=torch.float64) * kept[:, -1:]
        pick = torch.minimum(torch.searchsorted(kept, u, right=True), keep.sum(-1, keepdim=True) - 1)
        return order.gather(1, pick).view(-1).int()


def prepare(case, seed):
    x = _Inputs(seed)
    s = globals()["_prepare_" + case["kind"]](x, case)
    s["pkg"], s["case"] = x.pkg, case
    return s


def run(s):
    return globals()["_run_" + s["case"]["kind"]](s)


# ---------------------------------------------------------------------------------------------------------- decode
def _prepare_decode(x, c):
    b = c["batch"]
    wq, ws = x.fp8_weights(VOCAB, FP8_K)
    seeds, steps = x.addresses(b)
    return {"hidden": x.normal(b, FP8_K).to(torch.bfloat16), "w": wq, "w_scale": ws, "seeds": seeds, "steps": steps,
            "a": x.empty(b, FP8_K, dtype=torch.uint8), "a_scale": x.empty(b, FP8_K // 128, dtype=torch.float32),
            "logits": x.empty(b, VOCAB, dtype=torch.float32), "records": x.empty(b, 16, dtype=torch.uint8),
            "flag": torch.zeros(1, dtype=torch.int32, device=x.dev),
            "tokens": x.empty(b, dtype=torch.int32), "status": x.empty(b, dtype=torch.int32),
            "scratch": x.empty(x.pkg.sample_scratch_bytes(b, VOCAB), dtype=torch.uint8)}


def _run_decode(s):
    pkg, c = s["pkg"], s["case"]
    pkg.quantize_activations(s["hidden"], s["a"], s["a_scale"])
    pkg.head_fp8(s["a"], s["a_scale"], s["w"], s["w_scale"], s["logits"], s["flag"], row_extremes=s["records"])
    pkg.sample_logits(s["logits"], c["temperature"], c["top_p"], s["seeds"], s["steps"], tokens=s["tokens"],
                      status=s["status"], scratch=s["scratch"], row_extremes=s["records"])
    return {"tokens": s["tokens"], "status": s["status"], "logits": s["logits"], "flag": s["flag"]}


# ---------------------------------------------------------------------------------------------------------- sample
def _prepare_sample(x, c):
    seeds, steps = x.addresses(c["rows"])
    return {"logits": x.peaked_logits(c["rows"], c["vocab"]), "seeds": seeds, "steps": steps}


def _run_sample(s):
    c = s["case"]
    return s["pkg"].sample_logits(s["logits"], c["temperature"], c["top_p"], s["seeds"], s["steps"], top_k=c["top_k"])


# ---------------------------------------------------------------------------------------------------------- verify
def _prepare_verify(x, c):
    n, d, v = c["sequences"], c["drafts"], c["vocab"]
    target = x.peaked_logits(n * (d + 1), v)
    draft = target.view(n, d + 1, v)[:, :d].reshape(n * d, v) + DRAFT_NOISE * x.normal(n * d, v)
    seeds, steps = x.addresses(n)
    return {"target": target, "draft": draft, "ids": x.proposals(draft, c["temperature"], c["top_p"]), "seeds": seeds,
            "steps": steps, "scratch": x.empty(x.pkg.verify_scratch_bytes(n, d, v), dtype=torch.uint8),
            "results": x.empty(n * 40, dtype=torch.uint8), "status": x.empty(n, dtype=torch.int32)}


def _run_verify(s):
    c = s["case"]
    results, status = s["pkg"].verify_logits(s["target"], s["draft"], s["ids"], c["drafts"], c["temperature"], c["top_p"],
                                             s["seeds"], s["steps"], s["scratch"], s["results"], s["status"])
    return results.view(torch.int32), status


# ----------------------------------------------------------------------------------------------------- constrained
def _prepare_constrained(x, c):
    rows, n = c["rows"], c["history"]
    zipf = (1.0 / torch.arange(1, VOCAB + 1, device=x.dev, dtype=torch.float64) ** 1.1).cumsum(0)
    history = x.empty(rows, n, dtype=torch.int32)
    for r in range(rows):  # every conversation has its own Zipf distribution
        rank = torch.searchsorted(zipf, x.uniform(n, dtype=torch.float64) * zipf[-1])
        history[r] = torch.randperm(VOCAB, device=x.dev, generator=x.gen)[rank.clamp_(max=VOCAB - 1)].int()
    lens = torch.full((rows,), n, dtype=torch.int32, device=x.dev)
    if c["ragged"]:
        lens = (lens * (0.1 + 0.9 * x.uniform(rows))).int()
    mask = None
    if c["mask"]:  # 1-5 % of the ids, in runs of 8-263
        share = 0.01 + 0.04 * x.uniform(rows)
        most = int(0.05 * VOCAB / 136) + 1
        start = (x.uniform(rows, most) * (VOCAB - 300)).long()
        end = start + 8 + (x.uniform(rows, most) * 256).long()
        live = (torch.arange(most, device=x.dev) < (share * VOCAB / 136).clamp_min(1)[:, None]).int()
        edge = torch.zeros((rows, VOCAB + 1), dtype=torch.int32, device=x.dev)
        edge.scatter_add_(1, start, live).scatter_add_(1, end, -live)
        bits = (edge.cumsum(1)[:, :VOCAB] > 0).view(rows, VOCAB // 32, 32).long()
        words = (bits << torch.arange(32, device=x.dev)).sum(-1)
        mask = torch.where(words >= 2 ** 31, words - 2 ** 32, words).int()
    seeds, steps = x.addresses(rows)
    return {"logits": x.peaked_logits(rows, VOCAB), "history": history, "lens": lens, "mask": mask, "seeds": seeds,
            "steps": steps, "tokens": x.empty(rows, dtype=torch.int32), "status": x.empty(rows, dtype=torch.int32)}


def _run_constrained(s):
    c = s["case"]
    return s["pkg"].sample_logits(s["logits"], c["temperature"], c["top_p"], s["seeds"], s["steps"], top_k=c["top_k"],
                                  history=s["history"], history_len=s["lens"], repetition=1.1, presence=0.3,
                                  frequency=0.2, mask=s["mask"], tokens=s["tokens"], status=s["status"])


# ---------------------------------------------------------------------------------------------------------- engine
def _prepare_engine(x, c):
    d, k = c["drafts"], PLUGIN_K
    # logits of standard deviation 4 from normalised hidden states; the drafter sees almost the target's states
    w = x.weights(VOCAB, k, torch.bfloat16, 4.0 / math.sqrt(k))
    h = x.normal(d + 1, 4, k).to(torch.bfloat16)
    pre = 0.25 + 0.05 * x.normal(d + 1, 4)
    norm = (1.0 + 0.05 * x.normal(k)).to(torch.bfloat16)
    hidden = torch.einsum("mjk,mj->mk", h.float(), pre)
    hidden = hidden * torch.rsqrt(hidden.square().mean(-1, keepdim=True)) * norm.float()
    seeds, steps = x.addresses(1)
    rows = lambda m: x.empty(m, VOCAB, dtype=torch.float32)  # noqa: E731
    return {"h": h, "pre": pre, "norm": norm, "x_draft": (hidden[:d] + 0.03 * x.normal(d, k)).contiguous(),
            "w_target": w.float() if c["head"] == "f32" else w, "w_draft": w.clone(),
            "w_markov": x.weights(VOCAB, 256, torch.bfloat16, 0.01), "embedding": x.weights(VOCAB, 256, torch.bfloat16, 1.0),
            "last": torch.randint(0, VOCAB, (1,), device=x.dev, generator=x.gen), "seeds": seeds, "steps": steps,
            "x": x.empty(d + 1, k, dtype=torch.float32), "draft_rows": rows(d), "draft": rows(d), "target": rows(d + 1),
            "ids": x.empty(d, dtype=torch.int32), "ids_status": x.empty(d, dtype=torch.int32),
            "sample_scratch": x.empty(x.pkg.sample_scratch_bytes(1, VOCAB), dtype=torch.uint8),
            "verify_scratch": x.empty(x.pkg.verify_scratch_bytes(1, d, VOCAB), dtype=torch.uint8),
            "results": x.empty(40, dtype=torch.uint8), "status": x.empty(1, dtype=torch.int32)}


def _run_engine(s):
    pkg, c = s["pkg"], s["case"]
    d, t, top_p = c["drafts"], c["temperature"], c["top_p"]
    pkg.head_compact(s["x_draft"], s["w_draft"], s["draft_rows"])
    previous = s["last"]
    for k in range(d):  # a proposal is the Markov context of the next position
        pkg.markov_logits(s["draft_rows"][k], s["w_markov"], s["embedding"][previous].view(-1), s["draft"][k])
        pkg.sample_logits(s["draft"][k:k + 1], t, top_p, s["seeds"], s["steps"], slot=k, purpose=pkg.Purpose.Draft,
                          tokens=s["ids"][k:k + 1], status=s["ids_status"][k:k + 1], scratch=s["sample_scratch"])
        previous = s["ids"][k:k + 1]
    pkg.final_norm(s["h"], s["pre"], s["norm"], out=s["x"])
    if c["head"] == "f32":
        pkg.head_f32(s["x"], s["w_target"], s["target"])
    else:
        pkg.head_bf16(s["x"], s["w_target"], s["target"], decode_symbol=True)
    pkg.verify_logits(s["target"], s["draft"], s["ids"], d, t, top_p, s["seeds"], s["steps"], s["verify_scratch"],
                      s["results"], s["status"])
    return {"results": s["results"].view(torch.int32), "status": s["status"], "ids": s["ids"],
            "ids_status": s["ids_status"], "x": s["x"], "draft": s["draft"], "target": s["target"]}


# ----------------------------------------------------------------------------------------------------------- score
def _prepare_score(x, c):
    return {"logits": x.peaked_logits(c["rows"], c["vocab"])}


def _run_score(s):
    return s["pkg"].score_logits(s["logits"], s["case"]["top_n"])


# ------------------------------------------------------------------------------------------------------------ rows
def _prepare_rows(x, c):
    d, v = c["drafts"], c["vocab"]
    target = x.peaked_logits(d + 1, v)
    draft = target[:d] + DRAFT_NOISE * x.normal(d, v)
    seeds, steps = x.addresses(1)
    return {"target": target, "draft": draft, "ids": x.proposals(draft, c["temperature"], c["top_p"]), "seeds": seeds,
            "steps": steps}


def _run_rows(s):
    pkg, c = s["pkg"], s["case"]
    q, q_status = pkg.probabilities(s["draft"], c["temperature"], c["top_p"])
    p, p_status = pkg.probabilities(s["target"], c["temperature"], c["top_p"])
    results, status = pkg.verify_probabilities(s["ids"], q, p, c["drafts"], s["seeds"], s["steps"])
    return {"q": q, "p": p, "q_status": q_status, "p_status": p_status, "results": results.view(torch.int32),
            "status": status}


# ---------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Every input read once, every output written once; the multiply-adds of the heads."""
    c, kind = case, case["kind"]
    if kind == "decode":
        b = c["batch"]
        weights = VOCAB * FP8_K + 4 * (VOCAB // 128) * (FP8_K // 128)
        return {"bytes": weights + b * (2 * FP8_K + 4 * VOCAB + 24), "flops": 2.0 * b * VOCAB * FP8_K}
    if kind == "sample":
        return {"bytes": c["rows"] * (4 * c["vocab"] + 24), "flops": 0}
    if kind == "verify":
        rows = c["sequences"] * (2 * c["drafts"] + 1)
        return {"bytes": 4 * rows * c["vocab"] + c["sequences"] * (4 * c["drafts"] + 60), "flops": 0}
    if kind == "constrained":
        tokens = c["history"] * (0.55 if c["ragged"] else 1.0)  # a ragged batch fills 55 % of it on average
        return {"bytes": c["rows"] * (4 * VOCAB + 4 * tokens + (VOCAB // 8 if c["mask"] else 0) + 28), "flops": 0}
    if kind == "engine":
        d, k = c["drafts"], PLUGIN_K
        heads = VOCAB * k * (2 + (4 if c["head"] == "f32" else 2))
        return {"bytes": heads + 2 * 256 * VOCAB + 4 * VOCAB * (2 * d + 1) + 4 * k * d + 8 * k * (d + 1),
                "flops": 2.0 * VOCAB * k * (2 * d + 1)}
    if kind == "score":
        return {"bytes": c["rows"] * (4 * c["vocab"] + 12 * c["top_n"] + 16), "flops": 0}
    rows = 2 * c["drafts"] + 1
    return {"bytes": 12 * rows * c["vocab"], "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "decode":
        # fp32 sums of e4m3 products; a logit's last bits can move a draw that lies on the edge of two ids
        return {"rel": 1e-5, "differ": 0.005}
    if kind == "engine":
        # the BF16 heads have a fixed order of operations; the FP32 head's is free
        return {"rel": 2e-6} if case["head"] == "f32" else "exact"
    if kind == "score":
        return {"rel": 1e-12}
    if kind == "rows":
        return {"rel": 1e-13}  # fp64 rows whose sums have the reference's order: only exp() is free, in its last place
    return "exact"
