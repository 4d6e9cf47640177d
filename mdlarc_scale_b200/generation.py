"""Token generation with layered models: request scheduling over the slots of one session, and the command line.

    python -m mdlarc_scale_b200.generation --model DIR --prompts prompts.jsonl --max-new 64

Requests wait until a slot is free; the prompts of admitted requests are prefilled in packed calls of
bounded size (long prompts in portions) between runs of graph-replayed decode steps of the sequences already
generating; a finished sequence's slot goes to the next request.  Picking the next token (argmax or
temperature / top-k sampling) happens on the device.
"""
from __future__ import annotations

import argparse
import json
import sys
from collections import deque
from dataclasses import dataclass, field

import numpy as np
import torch

from .engine import EngineBase
from .inference import DEFAULT_PREFILL_TOKENS, POLL_EVERY
from .layered import Segment


@dataclass
class Request:
    rid: int
    prompt: list[int]
    fed: int = 0                 # prompt tokens already in the cache
    slot: int = -1
    produced: int = 0            # tokens picked so far (host count; an upper bound once the end token is out)
    output: list[int] = field(default_factory=list)
    tokens: np.ndarray | None = field(default=None, compare=False)     # the prompt as one array, from submit()


def _token_array(prompt) -> np.ndarray:
    try:
        tokens = np.array(prompt, np.int64)
        if tokens.ndim == 1:
            return tokens
    except (TypeError, ValueError, OverflowError, RuntimeError):
        pass
    return np.array([int(t) for t in prompt], object)     # elements that only int() understands, or refuses


class Scheduler:
    """Runs requests to completion on one session of a layered engine."""

    def __init__(self, engine: EngineBase, max_new: int, t_max: int, n_slots: int, prefill_tokens: int = DEFAULT_PREFILL_TOKENS,
                 end_token: int | None = None, temperature: float = 0.0, top_k: int | None = None, seed: int = 0,
                 want_logits: bool = False):
        self.engine, self.max_new = engine, int(max_new)
        self.end_token = -1 if end_token is None else int(end_token)
        self.session = engine.new_session(
            n_slots, t_max, self.max_new, min(prefill_tokens, n_slots * t_max), stop_on_end=True,
            want_step_logits=want_logits, temperature=temperature, top_k=top_k or 0, sample_seed=seed,
            sample_stream=np.zeros(n_slots, np.int64), end_token=self.end_token)
        self.waiting: deque[Request] = deque()
        self.filling: list[Request] = []
        self.decoding: list[Request] = []
        self.done: list[Request] = []
        self.step_logits: dict[int, torch.Tensor] = {}

    def submit(self, request: Request) -> None:
        n = len(request.prompt)
        if n == 0:
            raise ValueError("a prompt needs at least one token")
        if n + self.max_new - 1 > self.session.t_max:
            raise ValueError(f"prompt of {n} tokens plus {self.max_new} new ones exceeds the session's {self.session.t_max} positions")
        tokens = _token_array(request.prompt)
        if tokens.min() < 0 or tokens.max() >= self.engine.vocab_size:
            raise ValueError("a prompt token lies outside the vocabulary")
        request.tokens = tokens.astype(np.int64)
        self.waiting.append(request)

    # The device state of all admitted requests is set, and the results of all ended ones are read, together: with a few
    # launches and copies for each (35 to 90 us) the GPU waited 10 of 68 ms for the host at 150 requests.
    def _admit(self) -> None:
        admitted = []
        while self.waiting and self.session.free_slots:
            r = self.waiting.popleft()
            r.slot = self.session.acquire()
            admitted.append(r)
        if not admitted:
            return
        self.filling += admitted
        at = torch.tensor([[r.slot for r in admitted], [r.rid & 0x7FFFFFFF for r in admitted]]).to(self.engine.device, non_blocking=True)
        self.session.out_tokens.index_fill_(0, at[0], -1)
        self.session.sample_stream.index_copy_(0, at[0], at[1].to(torch.int32))

    def _prefill(self) -> None:
        room, call, armed = self.session.max_prefill_tokens, [], []
        for r in self.filling:
            n = min(room, len(r.tokens) - r.fed)
            if n <= 0:
                break
            last = r.fed + n == len(r.tokens)
            call.append(Segment(r.slot, r.tokens[r.fed:r.fed + n], arm=last))
            r.fed += n
            room -= n
            if last:
                armed.append(r)
        self.session.prefill_segments(call)
        for r in armed:
            self.filling.remove(r)
            r.produced = 1
            self.decoding.append(r)

    def _decode(self) -> None:
        left = min(self.max_new - r.produced for r in self.decoding)
        n = min(left, POLL_EVERY)
        if n > 0:
            self.session.decode(n)
            for r in self.decoding:
                r.produced += n
                self.session.lens[r.slot] += n

    def _retire(self) -> None:
        flags = self.session.finished() if self.end_token >= 0 else None
        ended = [r for r in self.decoding if r.produced >= self.max_new or (flags is not None and flags[r.slot])]
        if not ended:
            return
        if self.end_token < 0:      # all of them have max_new tokens: copied while the GPU is still at the last steps
            self._keep_logits(ended, [self.max_new] * len(ended))
        rows = self.session.out_tokens.cpu()
        for r in ended:
            row = rows[r.slot].tolist()
            if self.end_token in row:
                row = row[:row.index(self.end_token) + 1]
            r.output = row
        if self.end_token >= 0:
            self._keep_logits(ended, [len(r.output) for r in ended])
        gone = {id(r) for r in ended}
        self.decoding = [r for r in self.decoding if id(r) not in gone]
        for r in ended:
            self.session.release(r.slot)
            self.done.append(r)

    def _keep_logits(self, requests: list[Request], lengths: list[int]) -> None:
        """Each request's rows in memory of their own: one that is kept keeps no other's, nor rows it has not picked from."""
        if self.session.step_logits is None:
            return
        slots = self.session.step_logits.unbind(0)
        for r, n in zip(requests, lengths):
            self.step_logits[r.rid] = slots[r.slot].narrow(0, 0, n).clone()

    def run(self) -> list[Request]:
        """Until every submitted request is done; returns them in submission order."""
        while self.waiting or self.filling or self.decoding:
            self._admit()
            if self.filling:
                self._prefill()
            if self.decoding:
                self._decode()
                self._retire()
        self.session.poll()      # surfaces any device-side error word
        return sorted(self.done, key=lambda r: r.rid)

    def close(self) -> None:
        self.session.close()


def generate(engine: EngineBase, prompts, max_new: int, end_token: int | None = None, temperature: float = 0.0,
             top_k: int | None = None, seed: int = 0, max_batch: int = 256,
             prefill_tokens: int = DEFAULT_PREFILL_TOKENS, return_logits: bool = False):
    """Continuations of token-id prompts: one list of generated ids per prompt, the end token (if any) included.
    Greedy unless ``temperature > 0``; a request's random stream depends on ``seed`` and its index only."""
    if max_new <= 0 or not prompts:
        return ([[] for _ in prompts], {}) if return_logits else [[] for _ in prompts]
    t_max = max(len(p) for p in prompts) + max_new
    sched = Scheduler(engine, max_new, t_max, min(len(prompts), max_batch), prefill_tokens, end_token, temperature,
                      top_k, seed, return_logits)
    try:
        for i, p in enumerate(prompts):
            sched.submit(Request(i, p if isinstance(p, list) else [int(t) for t in p]))
        out = [r.output for r in sched.run()]
        return (out, sched.step_logits) if return_logits else out
    finally:
        sched.close()


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(description="generate token ids with a model folder (config.json + model.safetensors)")
    ap.add_argument("--model", required=True)
    ap.add_argument("--prompts", default="-", help="file of JSON lists of token ids, one a line ('-': standard input)")
    ap.add_argument("--max-new", type=int, default=64)
    ap.add_argument("--end-token", type=int, default=None)
    ap.add_argument("--dtype", default="bfloat16", help="bfloat16 | bfloat16-operands | float32")
    ap.add_argument("--temperature", type=float, default=0.0)
    ap.add_argument("--top-k", type=int, default=None)
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--max-batch", type=int, default=256)
    args = ap.parse_args(argv)
    from .registry import load_model
    engine = load_model(args.model, "cuda:0", args.dtype)
    src = sys.stdin if args.prompts == "-" else open(args.prompts)
    prompts = [json.loads(line) for line in src if line.strip()]
    for row in generate(engine, prompts, args.max_new, args.end_token, args.temperature, args.top_k, args.seed, args.max_batch):
        print(json.dumps(row))
    return 0


if __name__ == "__main__":
    sys.exit(main())
