"""Which form of a matrix-state recurrence a step of several tokens takes.

A walk (csrc/walk.cuh) spreads a head's columns over the chip and takes a sequence's tokens one after another: its time is the
longest sequence's chain, or the chip's share of all columns where they fill it, and two launches more than the block form.
The block form keeps a head in one block: a short prompt's tokens in one go, a longer one's in chunks side by side.  Neither is
better everywhere.  On a B200, microseconds of the block form and of the walk:

    matrix memory, 128 x 256:  one prompt of 2,048 tokens, 4 heads 186, 300;  8 heads 362, 315;  16 heads 734, 521
                               one prompt of 512 tokens, 4 heads 173, 81;     eight of 128 tokens, 8 heads 234, 108
                               32 prompts of 4 tokens, 8 heads 30, 47;        one of 4 tokens, 4 heads 15, 12
    matrix memory, 64 x 128:   one prompt of 1,024 tokens, 8 heads 97, 113;   8 prompts of 1,024, 8 heads 327, 279
    delta rule, 128 x 128:     one prompt of 2,048 tokens, 8 heads 608, 393;  of 8,192 tokens, 4 heads 1,178, 1,538
                               32 prompts of 4 tokens, 8 heads 19, 29;        32 of 64 tokens, 8 heads 150, 145

So both are estimated from the step's sizes and the walk is taken where it is at least a tenth faster.  The constants were fitted
to 4,300 measured steps (1 to 32 prompts of 4 to 8,192 tokens, 1 to 32 heads, key sizes 32, 64 and 128, value sizes 32 to 256);
of those three are more than 5 % slower than the block form (13 % at most), and one in thirteen more than 5 % slower than the
better of the two, most of them steps where the two are within a fifth of each other.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Callable

import torch

from ..kernels import ops

# the block form's chunks, and up to how many tokens it takes a sequence in one go (the delta rule's chain from chunk to chunk
# costs a product with a d x d matrix per chunk, so its chunks are longer)
MLSTM_CHUNK, MLSTM_WHOLE = 64, 128
DELTA_CHUNK, DELTA_WHOLE = 128, 128

# steps whose longest sequence brings fewer tokens stay with the block form: they are over before two more launches have paid
WALK_TOKENS = 4


@dataclass(frozen=True)
class Cost:
    """Constants of one recurrence, in microseconds (``d`` key size, ``dv`` value size, ``t`` threads of a block-form block)."""
    # the walk: launches; per eight heads (the kernels before and behind it take a token's heads eight at a time), with d and dv;
    start: float
    group: float
    group_d: float
    group_dv: float
    load: float                # a block's state in and out, per d and blocks an SM
    chain: float               # a token alone on an SM, and with d
    chain_d: float
    share: float               # a token, per block of the SM, and with d
    share_d: float
    extra_block: int           # column blocks beyond dv / 16
    # the block form: launch, and with t; a token alone, with t and d; a token per block of the SM, and with t
    first: float
    first_t: float
    token: float
    token_t: float
    token_d: float
    full: float
    full_t: float
    small: int                 # keys smaller than this keep less of an SM busy
    passes: float              # work of a chunk, in walks over its tokens; the chain from chunk to chunk, per chunk and d * d
    link: float
    link_dd: float


MLSTM = Cost(start=4.3, group=0.8, group_d=0.007, group_dv=0.02, load=0.006, chain=0.075, chain_d=0.0005, share=0.035, share_d=0.0005,
             extra_block=1, first=4.5, first_t=0.0024, token=0.76, token_t=0.0006, token_d=0.0025, full=0.0, full_t=0.0033, small=48,
             passes=1.6, link=0.1, link_dd=0.0)
DELTA = Cost(start=3.5, group=1.2, group_d=0.017, group_dv=0.005, load=0.008, chain=0.095, chain_d=0.0007, share=0.067, share_d=0.0007,
             extra_block=0, first=4.5, first_t=0.0036, token=1.0, token_t=0.0012, token_d=0.003, full=0.14, full_t=0.0043, small=16,
             passes=1.9, link=0.0, link_dd=0.00055)


def _either(a: float, b: float) -> float:
    """The larger of two bounds, a little more where they are close."""
    return (a ** 4 + b ** 4) ** 0.25


def estimates(cost: Cost, n_tokens: int, n_seqs: int, max_q: int, heads: int, d: int, dv: int, chunk: int, whole: int, sms: int) -> tuple:
    """(block form, walk) in microseconds; ``whole``: up to how many tokens the block form does not cut a prompt into chunks."""
    blocks = heads * n_seqs * (dv // 16 + cost.extra_block) / sms
    walk = (cost.start + -(-heads // 8) * (cost.group + cost.group_d * d + cost.group_dv * dv) + cost.load * d * blocks
            + max_q * _either(cost.chain + cost.chain_d * d, (cost.share + cost.share_d * d) * blocks))
    threads = (2 if d > 64 else 1) * max(d, dv)
    token = cost.token + cost.token_t * threads + cost.token_d * d
    full = cost.full + cost.full_t * threads * min(1.0, (d + 16) / (cost.small + 16))
    if max_q <= whole:
        per_sm = heads * n_seqs / sms
        if threads >= 512:       # an SM holds one such block
            per_sm = float(-(-heads * n_seqs // sms))
        block = cost.first + cost.first_t * threads + 0.0003 * d * dv * heads * n_seqs / sms + max_q * _either(token, full * per_sm)
    else:
        chunks = min(n_seqs * -(-max_q // chunk), n_tokens // chunk + n_seqs) * heads
        per_sm = float(-(-chunks // sms)) if threads >= 512 else chunks / sms
        block = cost.passes * chunk * _either(token, full * per_sm) + -(-max_q // chunk) * (cost.link + cost.link_dd * d * d)
    return block, walk


def takes_walk(cost: Cost, n_tokens: int, n_seqs: int, max_q: int, heads: int, d: int, dv: int, chunk: int, whole: int, sms: int) -> bool:
    """Whether a step takes the walk, for sizes that it has (the scratch sizes say so)."""
    if max_q < WALK_TOKENS:
        return False
    block, walk = estimates(cost, n_tokens, n_seqs, max_q, heads, d, dv, chunk, whole, sms)
    return walk < 0.9 * block


def run_mlstm(args: tuple, n_seqs: int, max_q: int, heads: int, d: int, dv: int, status: torch.Tensor,
              scratch: Callable[[str, int], torch.Tensor]) -> None:
    """A step of the matrix memory; ``args``: what ``ops.mlstm_walk`` and ``ops.mlstm_recurrence`` take in front of ``n_seqs``;
    ``scratch(name, floats)``: float32 scratch."""
    n = args[0].shape[0]
    walk = ops.mlstm_walk_scratch_floats(n, heads, d, dv)
    if walk and takes_walk(MLSTM, n, n_seqs, max_q, heads, d, dv, MLSTM_CHUNK, MLSTM_WHOLE, ops.sm_count(args[0].device)):
        ops.mlstm_walk(*args, n_seqs, heads, d, dv, status, scratch("mlstm.walk", walk))
        return
    chunk, max_chunks, area = 0, 1, None
    if max_q > MLSTM_WHOLE:
        chunk, max_chunks = MLSTM_CHUNK, -(-max_q // MLSTM_CHUNK)
        area = scratch("mlstm.scratch", ops.mlstm_scratch_floats(n_seqs, heads, d, dv, max_chunks))
    ops.mlstm_recurrence(*args, n_seqs, max_q, heads, d, dv, status, chunk, max_chunks, area)


def run_delta_rule(args: tuple, n_seqs: int, max_q: int, heads: int, kv_heads: int, d: int, dv: int, status: torch.Tensor,
                   scratch: Callable[[str, int], torch.Tensor], **form) -> None:
    """A step of the gated delta rule, as above; ``form``: ``head_decay`` and ``gate_silu``."""
    n = args[0].shape[0]
    walk = ops.delta_rule_walk_scratch_floats(n, heads, kv_heads, d, dv)
    if walk and takes_walk(DELTA, n, n_seqs, max_q, heads, d, dv, DELTA_CHUNK, DELTA_WHOLE, ops.sm_count(args[0].device)):
        ops.delta_rule_walk(*args, n_seqs, heads, kv_heads, d, dv, status, scratch("delta.walk", walk), **form)
        return
    chunk, max_chunks, area = 0, 1, None
    if max_q > DELTA_WHOLE:
        chunk, max_chunks = DELTA_CHUNK, -(-max_q // DELTA_CHUNK)
        area = scratch("delta.scratch", ops.delta_rule_scratch_floats(n_seqs, heads, d, dv, max_chunks))
    ops.delta_rule_recurrence(*args, n_seqs, max_q, heads, kv_heads, d, dv, status, chunk, max_chunks, area, **form)
