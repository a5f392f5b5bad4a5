"""Workloads of the library's public entry points, with the inputs a caller would have in hand.

One GPU plays one rank of an expert-parallel group of one: every expert is local, the sizes are
what one rank of a larger group sees (32 local experts of a DeepSeek-V3-like layer, 16 of a
Qwen3-30B-A3B-like one). Kinds:

    route    top-k routing of a batch of router logits
    a2a      dispatch -> combine with an identity expert in bf16 or fp16
    gemm     one expert GEMM (gate/up with SwiGLU and re-quantisation, or down) on ragged experts
    layer    the whole MoE layer: routing, dispatch with fp8 quantisation, both GEMMs, combine
    pages    KV-cache pages from one pool to another through the transfer engine, layer by layer
    rows     a column shard of a matrix written row by row into the wider matrix (TP reshard)
    encode   a batch of documents through the Unigram tokenizer (host memory, host threads)
"""

from __future__ import annotations

import base64
import functools
import json
import math
import threading
import weakref

import numpy as np
import torch

from pplx_garden.fabric_lib import PageIndices, TransferEngine
from pplx_garden.kernels.p2p_all_to_all import P2PAllToAll
from pplx_garden.models import ExpertParallelMoE, route_topk
from pplx_garden.ops import (
    MODE_BF16,
    MODE_SWIGLU_QUANT,
    grouped_fp8_gemm,
    quantize_1x128,
    quantize_128x128,
    topk_route,
)
from pplx_garden.unigram import Engine

PAGE_BYTES = 64 * 8 * 128 * 2  # 64 tokens x 8 KV heads x 128 dims, bf16
VOCAB_SIZE = 32000
LEXICON_SIZE = 50000
_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


def listed() -> list[dict]:
    return [
        # the router of one decode step: the smallest call there is, all latency and host path
        dict(name="route-decode", kind="route", tokens=128, experts=256, topk=8, dtype="fp32", bias=False),
        # the router of a large prefill batch, with the selection bias of load-balanced training
        dict(name="route-prefill", kind="route", tokens=32768, experts=256, topk=8, dtype="bf16", bias=True),
        # one decode step's dispatch and combine at the shape of the headline benchmark
        dict(name="a2a-decode", kind="a2a", tokens=128, capacity=128, hidden=7168, experts=256, topk=8,
             dtype="bf16", combine="per_route", split=False),
        # the same for a prefill chunk
        dict(name="a2a-prefill", kind="a2a", tokens=4096, capacity=4096, hidden=7168, experts=256, topk=8,
             dtype="bf16", combine="per_route", split=False),
        # expert up-projections of a Qwen3-like layer whose weights come with arbitrary fp32 scales
        dict(name="gemm-gate-up-fp32", kind="gemm", part="gate_up", hidden=2048, inter=768, experts=16,
             rows=16384, scales="fp32"),
        # expert down-projections of a DeepSeek-like layer with power-of-two scales
        dict(name="gemm-down-pow2", kind="gemm", part="down", hidden=7168, inter=2048, experts=8, rows=8192,
             scales="pow2"),
        # a decode step of a DeepSeek-like layer whose batch does not fill its capacity: bound by the weights
        dict(name="layer-decode", kind="layer", tokens=97, capacity=128, hidden=7168, inter=2048, experts=32,
             topk=8, routing="separate", fused_combine=False, scales="pow2"),
        # a Qwen3-like layer in prefill, routed inside the dispatch kernel
        dict(name="layer-prefill", kind="layer", tokens=2048, capacity=2048, hidden=2048, inter=768, experts=16,
             topk=8, routing="fused", fused_combine=False, scales="pow2"),
        # the largest: a DeepSeek-like layer on a prefill chunk, the down projection sending its rows itself
        dict(name="layer-long", kind="layer", tokens=4096, capacity=4096, hidden=7168, inter=2048, experts=32,
             topk=8, routing="separate", fused_combine=True, scales="pow2"),
        # prefill -> decode hand-over of one sequence of 19,000 tokens, four layers at a time
        dict(name="kv-pages", kind="pages", pages=297, layers=4),
        # one source shard of a tensor-parallel reshard, TP=8 -> TP=4, of a 7168 x 7168 bf16 matrix
        dict(name="reshard-rows", kind="rows", rows=7168, cols=896, slots=2),
        # the tokenizer on a corpus, eight threads
        dict(name="encode-corpus", kind="encode", docs=1024, chars=10000, threads=8),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _capacity(tokens: int) -> int:
    """What a server would size its context for: a power of two, at least 16."""
    return max(16, 1 << (tokens - 1).bit_length())


def draw(rng) -> dict:
    kind = rng.choice(["route", "route", "a2a", "a2a", "gemm", "gemm", "layer", "layer", "layer", "pages", "rows",
                       "encode"])
    if kind == "route":
        experts, topk = rng.choice([(64, 6), (128, 8), (160, 6), (256, 8), (384, 8), (512, 10)])
        return dict(kind=kind, tokens=_log_int(rng, 1, 32768), experts=experts, topk=topk,
                    dtype=rng.choice(["fp32", "bf16"]), bias=rng.random() < 0.5)
    if kind == "a2a":
        experts, topk = rng.choice([(16, 2), (32, 8), (64, 6), (128, 8), (256, 8)])
        tokens = _log_int(rng, 1, 4096)
        return dict(kind=kind, tokens=tokens, capacity=_capacity(tokens), hidden=rng.choice([1024, 2048, 4096, 7168]),
                    experts=experts, topk=topk, dtype=rng.choice(["bf16", "bf16", "fp16"]),
                    combine=rng.choice(["per_route", "per_route", "pre_reduce"]), split=rng.random() < 0.25)
    if kind == "gemm":
        hidden, inter, most_experts, most_rows = rng.choice([(2048, 768, 128, 32768), (7168, 2048, 32, 16384)])
        experts = _log_int(rng, 1, most_experts)
        return dict(kind=kind, part=rng.choice(["gate_up", "down"]), hidden=hidden, inter=inter, experts=experts,
                    rows=_log_int(rng, experts, most_rows), scales=rng.choice(["fp32", "pow2"]))
    if kind == "layer":
        hidden, inter, experts = rng.choice([(2048, 768, 16), (2048, 768, 64), (2048, 768, 128), (7168, 2048, 32)])
        tokens = _log_int(rng, 1, 4096)
        return dict(kind=kind, tokens=tokens, capacity=_capacity(tokens), hidden=hidden, inter=inter, experts=experts,
                    topk=8, routing=rng.choice(["separate", "fused"]), fused_combine=rng.random() < 0.4,
                    scales=rng.choice(["pow2", "pow2", "pow2", "fp32"]))
    if kind == "pages":
        return dict(kind=kind, pages=_log_int(rng, 1, 512), layers=rng.randint(1, 4))
    if kind == "rows":
        return dict(kind=kind, rows=_log_int(rng, 64, 7168), cols=8 * _log_int(rng, 4, 448), slots=rng.choice([2, 4]))
    return dict(kind=kind, docs=_log_int(rng, 1, 1024), chars=_log_int(rng, 200, 10000), threads=rng.choice([1, 8]))


def _device() -> torch.device:
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=_device()).manual_seed(seed)


def _router_logits(gen, tokens: int, experts: int, dtype=torch.float32) -> torch.Tensor:
    """N(0, 1) plus a per-expert N(0, 0.5): experts are not equally popular."""
    dev = _device()
    popularity = torch.randn(experts, generator=gen, device=dev) * 0.5
    return (torch.randn((tokens, experts), generator=gen, device=dev) + popularity).to(dtype)


def _routing(logits: torch.Tensor, topk: int) -> tuple[torch.Tensor, torch.Tensor]:
    top = torch.topk(logits, topk, dim=-1)
    return top.indices.to(torch.int32).view(torch.uint32), torch.softmax(top.values, dim=-1)


# ---- route ----


def _prepare_route(case: dict, seed: int) -> dict:
    gen = _gen(seed)
    bias = torch.randn(case["experts"], generator=gen, device=_device()) * 0.1 if case["bias"] else None
    return dict(logits=_router_logits(gen, case["tokens"], case["experts"], _DTYPES[case["dtype"]]), bias=bias)


def _run_route(case: dict, s: dict):
    return topk_route(s["logits"], case["topk"], s["bias"])


# ---- a2a ----


class _Owned:
    """Destroys what it holds when the state goes away, as a caller does at shutdown."""

    def __init__(self, thing) -> None:
        self.thing = thing

    def __del__(self) -> None:
        self.thing.destroy()


def _prepare_a2a(case: dict, seed: int) -> dict:
    gen, dev, dtype = _gen(seed), _device(), _DTYPES[case["dtype"]]
    T, H = case["tokens"], case["hidden"]
    a2a = P2PAllToAll(
        max_num_tokens=case["capacity"], num_experts=case["experts"], expert_padding=1, hidden_dim=H,
        hidden_dim_scale=None, in_dtype=dtype, out_dtype=dtype, scale_dtype=None,
        num_experts_per_token=case["topk"], device=dev, dp_group=None, global_group=None,
        combine_mode=case["combine"])
    indices, weights = _routing(_router_logits(gen, T, case["experts"]), case["topk"])
    return dict(
        owner=_Owned(a2a), indices=indices, weights=weights,
        x=torch.randn((T, H), generator=gen, device=dev).to(dtype),
        num=torch.zeros(case["experts"], dtype=torch.int32, device=dev),
        expert_x=torch.zeros((a2a.max_recv_rows, H), dtype=dtype, device=dev),
        out=torch.zeros((T, H), dtype=dtype, device=dev))


def _run_a2a(case: dict, s: dict):
    # the rows of an expert have no defined order, so they are not an output here; the identity
    # expert hands them to combine, whose result depends on every one of them
    a2a, num, rows, out, idx, w = s["owner"].thing, s["num"], s["expert_x"], s["out"], s["indices"], s["weights"]
    if case["split"]:
        a2a.dispatch(num, rows, None, s["x"], None, idx, w, do_recv=False)
        a2a.dispatch(num, rows, None, s["x"], None, idx, w, do_send=False)
        a2a.combine(out, idx, w, rows, do_recv=False)
        a2a.combine(out, idx, w, rows, do_send=False)
    else:
        a2a.dispatch(num, rows, None, s["x"], None, idx, w)
        a2a.combine(out, idx, w, rows)
    return num, out


# ---- gemm ----


def _ragged_counts(seed: int, experts: int, rows: int) -> np.ndarray:
    """Rows per expert of a router whose experts are not equally popular; they add up to `rows`."""
    rng = np.random.default_rng(seed)
    share = rng.dirichlet(np.full(experts, 8.0))
    return rng.multinomial(rows, share)


def _fp8_zeros(*shape: int) -> torch.Tensor:
    return torch.zeros(shape, dtype=torch.uint8, device=_device()).view(torch.float8_e4m3fn)


def _prepare_gemm(case: dict, seed: int) -> dict:
    gen, dev = _gen(seed), _device()
    E, R, H, I, pow2 = case["experts"], case["rows"], case["hidden"], case["inter"], case["scales"] == "pow2"
    n, k = (2 * I, H) if case["part"] == "gate_up" else (H, I)
    a, a_scale = quantize_1x128(torch.randn((R, k), generator=gen, device=dev), pow2=pow2)
    b, b_scale = quantize_128x128(torch.randn((E, n, k), generator=gen, device=dev) * k ** -0.5, pow2=pow2)
    s = dict(a=a, a_scale=a_scale, b=b, b_scale=b_scale, error=torch.zeros(1, dtype=torch.int32, device=dev),
             counts=torch.tensor(_ragged_counts(seed, E, R), dtype=torch.int32, device=dev))
    if case["part"] == "gate_up":
        s.update(out=_fp8_zeros(R, I), out_scale=torch.zeros((R, I // 128), dtype=torch.float32, device=dev))
    else:
        s.update(out=torch.zeros((R, H), dtype=torch.bfloat16, device=dev), out_scale=None)
    return s


def _run_gemm(case: dict, s: dict):
    grouped_fp8_gemm(s["a"], s["a_scale"], s["b"], s["b_scale"], s["counts"], s["out"], s["out_scale"],
                     mode=MODE_SWIGLU_QUANT if case["part"] == "gate_up" else MODE_BF16, error_flag=s["error"],
                     scale_format=case["scales"])
    return s["out"], s["out_scale"], s["error"]


# ---- layer ----


def _prepare_layer(case: dict, seed: int) -> dict:
    gen, dev = _gen(seed), _device()
    T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
    w13 = torch.randn((E, 2 * I, H), generator=gen, device=dev) * 0.02
    w2 = torch.randn((E, H, I), generator=gen, device=dev) * 0.02
    layer = ExpertParallelMoE(
        hidden_dim=H, intermediate_dim=I, num_experts=E, num_experts_per_token=K, max_num_tokens=case["capacity"],
        device=dev, global_group=None, w13=w13, w2=w2, fused_combine=case["fused_combine"],
        scale_format=case["scales"])
    return dict(
        owner=_Owned(layer), logits=_router_logits(gen, T, E),
        x=torch.randn((T, H), generator=gen, device=dev).to(torch.bfloat16),
        indices=torch.zeros((T, K), dtype=torch.int32, device=dev).view(torch.uint32),
        weights=torch.zeros((T, K), dtype=torch.float32, device=dev))


def _run_layer(case: dict, s: dict):
    layer = s["owner"].thing
    if case["routing"] == "fused":
        indices, weights = s["indices"], s["weights"]
        y = layer(s["x"], indices, weights, logits=s["logits"])
    else:
        indices, weights = route_topk(s["logits"], case["topk"])
        y = layer(s["x"], indices, weights)
    return y, indices, weights


# ---- pages, rows ----


class _Link:
    """A sending and a receiving engine on one GPU; stopped when the last user is gone."""

    def __init__(self) -> None:
        device = torch.cuda.current_device()
        self.tx, self.rx = TransferEngine(1, [device]), TransferEngine(1, [device])
        self.imm = 0x1000

    def __del__(self) -> None:
        self.tx.stop()
        self.rx.stop()


_link_ref = None


def _link() -> _Link:
    global _link_ref
    link = _link_ref() if _link_ref is not None else None
    if link is None:
        link = _Link()
        _link_ref = weakref.ref(link)
    return link


class _Registered:
    """A source and a destination tensor, registered with the two engines while the state lives."""

    def __init__(self, src: torch.Tensor, dst: torch.Tensor) -> None:
        self.link, self.src, self.dst = _link(), src, dst
        torch.cuda.synchronize()
        self.handle, _ = self.link.tx.register_tensor(src)
        _, self.desc = self.link.rx.register_tensor(dst)

    def __del__(self) -> None:
        self.link.tx.unregister_memory(self.src.data_ptr())
        self.link.rx.unregister_memory(self.dst.data_ptr())


class _Completions:
    """Counts the transfers of one pass; wait() returns when all of them are through."""

    def __init__(self, count: int) -> None:
        self.errors: list[str] = []
        self.count = count
        self.sem = threading.Semaphore(0)

    def done(self) -> None:
        self.sem.release()

    def error(self, message: str) -> None:
        self.errors.append(message)
        self.sem.release()

    def wait(self) -> None:
        for _ in range(self.count):
            if not self.sem.acquire(timeout=60):
                raise RuntimeError("a transfer did not complete")
        if self.errors:
            raise RuntimeError(self.errors[0])


def _prepare_pages(case: dict, seed: int) -> dict:
    gen, n, layers = _gen(seed), case["pages"], case["layers"]
    rng = np.random.default_rng(seed)
    pool = 2 * n * layers
    src = torch.randint(0, 256, (pool, PAGE_BYTES), generator=gen, device=_device(), dtype=torch.uint8)
    dst = torch.zeros((pool, PAGE_BYTES), dtype=torch.uint8, device=_device())
    plan = []
    src_order, dst_order = rng.permutation(pool), rng.permutation(pool)
    for i in range(layers):
        plan.append((PageIndices(src_order[i * n:(i + 1) * n].tolist()),
                     PageIndices(dst_order[i * n:(i + 1) * n].tolist())))
    return dict(mem=_Registered(src, dst), plan=plan)


def _run_pages(case: dict, s: dict):
    mem, link, n = s["mem"], s["mem"].link, case["pages"]
    # every layer is sent and, on the receiving side, announced: two completions each
    all_done = _Completions(2 * len(s["plan"]))
    for src_pages, dst_pages in s["plan"]:
        link.imm += 1
        link.rx.set_imm_count_expected(link.imm, n, all_done.done)
        link.tx.submit_paged_writes(PAGE_BYTES, mem.handle, src_pages, PAGE_BYTES, 0, mem.desc, dst_pages, PAGE_BYTES, 0,
                                    link.imm, all_done.done, all_done.error)
    all_done.wait()
    return mem.dst


def _prepare_rows(case: dict, seed: int) -> dict:
    gen, R, C, slots = _gen(seed), case["rows"], case["cols"], case["slots"]
    src = torch.randn((R, C), generator=gen, device=_device()).to(torch.bfloat16)
    dst = torch.zeros((R, C * slots), dtype=torch.bfloat16, device=_device())
    return dict(mem=_Registered(src, dst), pages=PageIndices(list(range(R))))


def _run_rows(case: dict, s: dict):
    mem, row_bytes = s["mem"], 2 * case["cols"]
    done = _Completions(1)
    # "page" r is row r of the matrix; the shard fills the last of the destination's column slots
    mem.link.tx.submit_paged_writes(row_bytes, mem.handle, s["pages"], row_bytes, 0, mem.desc, s["pages"],
                                    case["slots"] * row_bytes, (case["slots"] - 1) * row_bytes, None, done.done, done.error)
    done.wait()
    return mem.dst


# ---- encode ----


@functools.lru_cache(maxsize=1)
def _tokenizer() -> str:
    """A Unigram tokenizer.json of 32,000 pieces with Zipf(1.1) scores and an empty charsmap."""
    rng = np.random.default_rng(0)
    letters = np.array(list("abcdefghijklmnopqrstuvwxyz"))
    pieces = dict.fromkeys([f"<0x{i:02X}>" for i in range(256)] + list("▁abcdefghijklmnopqrstuvwxyzéü"))
    while len(pieces) < VOCAB_SIZE:
        body = "".join(rng.choice(letters, rng.integers(1, 13)))
        pieces["▁" + body if rng.random() < 0.5 else body] = None
    mass = rng.permutation(np.arange(1, VOCAB_SIZE + 1)) ** -1.1
    scores = np.log(mass / mass.sum())
    metaspace = {"type": "Metaspace", "replacement": "▁", "prepend_scheme": "always", "split": True}
    charsmap = base64.b64encode(bytes(4)).decode()
    return json.dumps({
        "version": "1.0", "added_tokens": [],
        "normalizer": {"type": "Precompiled", "precompiled_charsmap": charsmap},
        "pre_tokenizer": metaspace, "decoder": metaspace,
        "model": {"type": "Unigram", "unk_id": 0, "byte_fallback": False,
                  "vocab": [[p, float(s)] for p, s in zip(pieces, scores)]}})


@functools.lru_cache(maxsize=1)
def _lexicon() -> np.ndarray:
    """50,000 words of 2 to 10 letters, some with an accented one."""
    rng = np.random.default_rng(1)
    letters = np.array(list("abcdefghijklmnopqrstuvwxyz" * 8 + "éü"))
    sizes = rng.integers(2, 11, LEXICON_SIZE)
    stream = "".join(rng.choice(letters, int(sizes.sum())))
    ends = np.cumsum(sizes)
    return np.array([stream[e - n:e] for e, n in zip(ends.tolist(), sizes.tolist())], dtype=object)


def _prepare_encode(case: dict, seed: int) -> dict:
    # Words drawn Zipf(1.1) from the lexicon, about seven characters each with the space. The seed
    # orders them: another seed gives other documents with as many tokens in all.
    mass = np.arange(1, LEXICON_SIZE + 1) ** -1.1
    per_doc = max(1, case["chars"] // 7)
    words = np.random.default_rng(2).choice(LEXICON_SIZE, case["docs"] * per_doc, p=mass / mass.sum())
    words = np.random.default_rng(seed).permutation(words).reshape(case["docs"], per_doc)
    docs = [" ".join(row) for row in _lexicon()[words].tolist()]
    return dict(engine=Engine.from_hf_json_bytes(_tokenizer()), docs=docs)


def _run_encode(case: dict, s: dict):
    return s["engine"].encode_batch_flat(s["docs"], case["threads"])


# ---- the interface ----

_PREPARE = dict(route=_prepare_route, a2a=_prepare_a2a, gemm=_prepare_gemm, layer=_prepare_layer, pages=_prepare_pages,
                rows=_prepare_rows, encode=_prepare_encode)
_RUN = dict(route=_run_route, a2a=_run_a2a, gemm=_run_gemm, layer=_run_layer, pages=_run_pages, rows=_run_rows,
            encode=_run_encode)


def prepare(case: dict, seed: int):
    return case, _PREPARE[case["kind"]](case, seed)


def run(state):
    case, s = state
    return _RUN[case["kind"]](case, s)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "route":
        T, E, K = case["tokens"], case["experts"], case["topk"]
        return dict(bytes=T * E * (4 if case["dtype"] == "fp32" else 2) + 8 * T * K + (4 * E if case["bias"] else 0),
                    flops=0)
    if kind == "a2a":
        # tokens in, expert rows out and in again, tokens out, the routing table twice
        T, K, H = case["tokens"], case["topk"], case["hidden"]
        return dict(bytes=2 * H * (2 * T + 2 * T * K) + 16 * T * K + 4 * case["experts"], flops=2 * T * K * H)
    if kind == "gemm":
        E, R, H, I = (case[k] for k in ("experts", "rows", "hidden", "inter"))
        n, k = (2 * I, H) if case["part"] == "gate_up" else (H, I)
        out = R * I + R * I // 32 if case["part"] == "gate_up" else 2 * R * H
        return dict(bytes=R * k + R * k // 32 + E * n * k + E * n * k // 4096 + 4 * E + out, flops=2 * R * n * k)
    if kind == "layer":
        T, H, I, E, K = (case[k] for k in ("tokens", "hidden", "inter", "experts", "topk"))
        experts_hit = E * (1 - (1 - K / E) ** T)
        return dict(bytes=4 * T * H + 4 * T * E + 8 * T * K + experts_hit * 3 * H * I * (1 + 1 / 4096),
                    flops=2 * T * K * 3 * H * I)
    if kind == "pages":
        return dict(bytes=2 * case["pages"] * case["layers"] * PAGE_BYTES, flops=0)
    if kind == "rows":
        return dict(bytes=4 * case["rows"] * case["cols"], flops=0)
    # text in, about one int32 token id per 2.5 characters out
    return dict(bytes=int(case["docs"] * case["chars"] * 2.6), flops=0)


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("pages", "rows", "encode"):
        return "exact"
    if kind == "route":
        return dict(rel=1e-5, max=1e-4)
    if kind == "gemm" and case["part"] == "gate_up":
        # e4m3 results: a sum that rounds the other way moves a value by an eighth of itself, and a
        # row maximum at the edge of a power of two moves a block's scale by a factor of two
        return dict(rel=1e-2, max=0.99)
    # bf16 and fp16 results; in the layer an e4m3 rounding inside may go the other way too
    return dict(rel=1e-2)
