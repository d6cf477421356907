"""CPU ORACLE (test infrastructure, not product code) - pure-Python restatement of the reference's greedy Jacobi
decoding state machines.  Only tests/, __graft_entry__.smoke() and bench.py's cpu_baseline/reference arm may import
this module; the product path (jacobiforcing_b200/) never does.

Every function restates one reference function and cites it (paths within the reference):

  hf_prefill            modeling/cllm2_qwen2_modeling_kv_terminate_on_eos_improved_multiblock_lookahead_unified.py:175-225
  hf_single_block       modeling/cllm2_qwen2_modeling_kv_terminate_on_eos_improved.py:140-276
  hf_multiblock         modeling/..._multiblock_lookahead_unified.py:230-740   (helpers :62-91, :264-271, :317-377, :387-411)
  hf_driver             JacobiForcing/jacobi_forcing_inference_MR_humaneval.py:152-250
  engine_fixed_len      inference_engine/engine/jacobi_decoding.py:303-445 (single), :448-724 (batched)

The model is reached only through a small "forward" object mirroring what the reference does to its DynamicCache:

  fwd.kv_len()            -> int                      past_key_values.get_seq_length()
  fwd.forward(rows)       -> greedy[B][L]             one forward over rows at positions kv_len+arange(L); every row's
                                                      K/V is appended (DynamicCache.update), so kv_len grows by L and the
                                                      cache batch becomes B (_resize_dynamic_cache_batch, :93-127)
  fwd.select_row(r)       -> None                     keep cache row r only (:500-502)
  fwd.trim(n)             -> None                     delete_false_key_value(n) (:36-59); n <= 0 is a no-op

greedy[b][j] = argmax of the logits at position j of row b (first index wins ties, torch.argmax on CPU).
Pinned against the unmodified reference: tests/golden/*.json (generated by oracle/make_golden.py).
"""
from __future__ import annotations

import math
from collections import deque
from dataclasses import dataclass, field
from typing import Callable, List, Optional, Sequence


# --------------------------------------------------------------------------------------------------------------
# traces
# --------------------------------------------------------------------------------------------------------------
@dataclass
class Trace:
    """Per-forward record: what `out` looked like (the reference feeds exactly this tensor to embed_tokens)."""
    rows: List[List[List[int]]] = field(default_factory=list)   # per forward: B rows of L tokens
    kv_before: List[int] = field(default_factory=list)

    def log(self, kv: int, rows: Sequence[Sequence[int]]) -> None:
        self.kv_before.append(int(kv))
        self.rows.append([list(map(int, r)) for r in rows])


def _leading_matches(draft_tail: Sequence[int], greedy_head: Sequence[int]) -> int:
    """(mismatch.cumsum(-1) == 0).sum(-1) for mismatch = draft[1:] != greedy[:-1]."""
    k = 0
    for d, g in zip(draft_tail, greedy_head):
        if d != g:
            break
        k += 1
    return k


# --------------------------------------------------------------------------------------------------------------
# prefill (unified.py:175-225; identical in improved.py:68-138)
# --------------------------------------------------------------------------------------------------------------
def hf_prefill(fwd, prompt: Sequence[int], draft: Sequence[int], trace: Optional[Trace] = None):
    """Forward prompt ++ n draft tokens; prefill_drafted_n_gram = argmax(logits[:, -n-1:-1]); crop KV by n.
    Returns (first_correct_token, prefill_drafted_n_gram)."""
    n = len(draft)
    assert fwd.kv_len() == 0
    row = list(prompt) + list(draft)
    if trace is not None:
        trace.log(0, [row])
    greedy = fwd.forward([row])[0]
    fwd.select_row(0)
    drafted = [int(t) for t in greedy[len(row) - n - 1: len(row) - 1]]
    if n > 0:
        fwd.trim(n)                                       # :222-223
    return drafted[0], drafted


# --------------------------------------------------------------------------------------------------------------
# single-block greedy Jacobi (improved.py:140-276): the draft shrinks by the accepted count every iteration
# --------------------------------------------------------------------------------------------------------------
def hf_single_block(fwd, input_ids: Sequence[int], n: int, eos: Optional[int] = None,
                    trace: Optional[Trace] = None):
    """Returns (next_token, accepted[<= n], iters)."""
    out = [int(t) for t in input_ids]
    accepted_n_gram: List[int] = []
    total_accepted = 0
    itr = 0
    next_token = None
    while total_accepted < n:                              # :150
        itr += 1
        if trace is not None:
            trace.log(fwd.kv_len(), [out])
        greedy_full = fwd.forward([out])[0]                # logits for all L positions
        fwd.select_row(0)
        L = len(out)
        greedy_tokens = greedy_full[:-1]                   # :197
        raw = _leading_matches(out[1:], greedy_tokens) + 1  # :199-202
        num_accepted = raw
        if eos is not None and eos in out[:raw]:           # :206-211
            num_accepted = out[:raw].index(eos) + 1
        accepted_n_gram.extend(out[:num_accepted])         # :214-216
        total_accepted += num_accepted
        if eos is not None and eos in out[:num_accepted]:  # :219-227 (KV left in the reference's odd trimmed state)
            return eos, accepted_n_gram[:total_accepted], itr
        if raw < L:                                        # :231-255 rejected tail
            fwd.trim(L - raw)                              # :233
            next_token = int(greedy_full[raw - 1])         # :235
            if eos is not None and next_token == eos:      # :238-247
                accepted_n_gram.append(next_token)
                total_accepted += 1
                return next_token, accepted_n_gram[:total_accepted], itr
            out = [next_token] + [int(t) for t in greedy_full[raw:L - 1]]   # :250-255
        else:                                              # :258-273 everything accepted
            next_token = int(greedy_full[-1])
            total_accepted += 1                            # the write at index n is a silent no-op on a width-n tensor
            if eos is not None and next_token == eos:
                return next_token, accepted_n_gram[:n], itr
    return next_token, accepted_n_gram[:n], itr            # :276


# --------------------------------------------------------------------------------------------------------------
# multiblock + rejection recycling (unified.py:230-740)
# --------------------------------------------------------------------------------------------------------------
def _build_candidates(pool: deque, token_val: int, out_row: Sequence[int]) -> List[List[int]]:
    """unified.py:62-91 with nearest=False: newest -> oldest, skipping the very last pool entry."""
    cands: List[List[int]] = []
    L_out = len(out_row)
    for seq in reversed(list(pool)[:-1]):
        if token_val in seq:
            pos = seq.index(token_val)
            cand = list(seq[pos:])
            if len(cand) > L_out:
                cand = cand[:L_out]
            elif len(cand) < L_out:
                cand = cand + list(out_row[len(cand):L_out])
            cands.append(cand)
    return cands


def _ensure_rows(rows: List[List[int]], B: int) -> List[List[int]]:
    """_ensure_batch_like_ra (:288-312): broadcast / tile-and-slice a block's rows to B rows."""
    if len(rows) == 0 or len(rows[0]) == 0:
        return [[] for _ in range(B)]
    if len(rows) == B:
        return rows
    if len(rows) == 1:
        return [list(rows[0]) for _ in range(B)]
    reps = (B + len(rows) - 1) // len(rows)
    return [list(r) for r in (rows * reps)[:B]]


def hf_multiblock(fwd, input_ids: Sequence[int], n: int, K: int = 2, r: float = 0.85,
                  lookahead_start_ratio: float = 0.0, n_gram_pool_size: int = 4, eos: Optional[int] = None,
                  pad: Optional[int] = None, max_iteration_count: int = 128, trace: Optional[Trace] = None):
    """Returns (next_token or None, accepted tokens, iters).  `num_blocks`, `active_blocks` and the list index
    space are three separate things, exactly as in the reference."""
    pool: deque = deque(maxlen=n_gram_pool_size)           # :238
    out_acc: List[List[int]] = [[]]                        # :249  accepted prefix per block (always one row)
    q_draft: List[List[List[int]]] = [[[int(t) for t in input_ids]]]   # :252 rows x L per block
    need_reverify = [False]
    total_acc = [0]
    num_blocks = 1
    active_blocks = 1
    RA = 0
    last_next_token: Optional[int] = None                  # :259 (an empty [1,0] tensor in the reference)
    prompt_len = fwd.kv_len()                              # :261
    spawn_threshold = math.ceil(r * n)                     # :262

    def committed_len(cur_RA: int) -> int:                 # :264-271
        c = prompt_len
        for b in range(num_blocks):
            if b != cur_RA and not need_reverify[b]:
                c += len(out_acc[b])
        return c + len(out_acc[cur_RA])

    def final_ret() -> List[int]:                          # :533-537, :602-606, :725-730
        ret: List[int] = []
        for bb in range(num_blocks):
            if bb != RA and not need_reverify[bb] and len(out_acc[bb]) > 0:
                ret.extend(out_acc[bb])
        ret.extend(out_acc[RA])
        return ret

    def concat_all_blocks_seq() -> List[int]:              # :387-411 (first row of every block, pads stripped)
        seq: List[int] = []
        for bb in range(num_blocks):
            seq.extend(out_acc[bb])
            if len(q_draft[bb]) > 0 and len(q_draft[bb][0]) > 0:
                seq.extend(q_draft[bb][0])
        if pad is not None:
            seq = [t for t in seq if t != pad]
        return seq

    iters = 0
    while iters < max_iteration_count:                     # :414
        iters += 1
        # ---- build_out_and_spans (:317-377); cursor starts at 1 so logits[start-1 : start-1+L] are the span's own
        B_ra = len(q_draft[RA])
        pieces: List[List[List[int]]] = []
        spans = []
        cursor = 1
        L_ra = len(q_draft[RA][0]) if B_ra > 0 else 0
        if L_ra > 0:
            pieces.append(q_draft[RA])
            spans.append((RA, cursor, L_ra))
            cursor += L_ra
        for b in range(num_blocks):
            if b == RA or not need_reverify[b]:
                continue
            if len(out_acc[b]) > 0:
                pieces.append(_ensure_rows([out_acc[b]], B_ra))
                cursor += len(out_acc[b])
            L_tail = len(q_draft[b][0]) if len(q_draft[b]) > 0 else 0
            if L_tail > 0:
                pieces.append(_ensure_rows(q_draft[b], B_ra))
                spans.append((b, cursor, L_tail))
                cursor += L_tail
        if not pieces:                                     # :418-419
            break
        out_rows = [sum((p[i] for p in pieces), []) for i in range(B_ra)]
        if len(out_rows) == 0 or len(out_rows[0]) == 0:
            break
        if trace is not None:
            trace.log(fwd.kv_len(), out_rows)
        greedy_all = fwd.forward(out_rows)                 # :429-463
        B_out = len(out_rows)

        for (b, start, L) in spans:                        # :467
            block_greedy = [g[start - 1:start - 1 + L] for g in greedy_all]          # :473-476
            draft_rows = q_draft[b]
            B_b = len(draft_rows)
            nrows = max(B_b, B_out)
            if B_b not in (1, nrows) or B_out not in (1, nrows):
                raise RuntimeError("reference would fail to broadcast draft rows against greedy rows")
            accepted = []
            for i in range(nrows):                         # :482-486
                d = draft_rows[i if B_b > 1 else 0]
                g = block_greedy[i if B_out > 1 else 0]
                accepted.append(_leading_matches(d[1:], g[:-1]) + 1)
            best_idx = accepted.index(max(accepted)) if b == RA else 0               # :487-491
            acc_len_raw = accepted[best_idx]
            draft = list(draft_rows[best_idx]) if best_idx < B_b else []             # :496
            greedy = [int(t) for t in block_greedy[best_idx]]                        # :499
            fwd.select_row(best_idx)                                                 # :500-502
            L_eff = len(draft)
            if L_eff == 0:
                continue
            acc_len = acc_len_raw
            eos_reached = False
            if eos is not None and b == RA and acc_len > 0 and eos in draft[:acc_len]:   # :514-521
                acc_len = draft[:acc_len].index(eos) + 1
                eos_reached = True
            has_rejected = acc_len < L_eff                                           # :523
            if acc_len > 0:                                                          # :526-528
                out_acc[b] = out_acc[b] + draft[:acc_len]
                total_acc[b] += acc_len
            if eos_reached and b == RA:                                              # :531-547
                ret = final_ret()
                fwd.trim(fwd.kv_len() - (prompt_len + len(ret)))
                return draft[acc_len - 1], ret, iters
            if has_rejected:                                                         # :550-588
                nxt = greedy[max(acc_len - 1, 0)]
                q_draft[b] = [[nxt] + greedy[acc_len:L_eff - 1]]
                if b == RA:
                    concat_seq = concat_all_blocks_seq()
                    if len(concat_seq) > 0:
                        pool.append(concat_seq)
                    tail = greedy[acc_len:L_eff - 1]
                    if len(tail) > 0:
                        pool.append(tail)
                if b == RA and (total_acc[b] / n >= lookahead_start_ratio):
                    cands = _build_candidates(pool, nxt, q_draft[b][0])
                    if len(cands) > 1:                                               # :579
                        q_draft[b] = [q_draft[b][0]] + cands
            else:                                                                    # :590-593
                q_draft[b] = [[]]
                nxt = greedy[-1]
            if b == RA:
                last_next_token = nxt
            if eos is not None and b == RA and last_next_token == eos:               # :599-614
                out_acc[b] = out_acc[b] + [last_next_token]
                ret = final_ret()
                fwd.trim(fwd.kv_len() - (prompt_len + len(ret)))
                return last_next_token, ret, iters

        fwd.trim(fwd.kv_len() - committed_len(RA))                                   # :617-626

        newest_id = num_blocks - 1                                                   # :629-653 spawn
        if total_acc[newest_id] >= spawn_threshold and active_blocks < K:
            if pad is None:
                raise ValueError("pad_token_id must be provided when spawning pseudo-active blocks.")
            ra_rows = q_draft[RA]
            L_cur = len(ra_rows[0]) if len(ra_rows) > 0 else 0
            pad_len = max(0, n - L_cur)
            q_draft.append([list(row) + [pad] * pad_len for row in ra_rows])
            out_acc.append([])
            total_acc.append(0)
            need_reverify.append(True)
            num_blocks += 1
            active_blocks += 1

        if total_acc[RA] >= n:                                                       # :656-716 promote
            for b in range(num_blocks):
                if need_reverify[b] and total_acc[b] > 0:
                    q_full = out_acc[b] + list(q_draft[b][0])
                    assert len(q_full) == n, f"draft size mismatch: draft at {len(q_full)} vs. n_token_seq_len {n}"
                    out_acc[b] = []
                    total_acc[b] = 0
                    q_draft[b] = [[last_next_token] + q_full[1:]]
                    need_reverify[b] = False
                    RA = b
                    fwd.trim(fwd.kv_len() - committed_len(RA))
                    active_blocks -= 1
                    num_blocks -= 1
                    break
                active_blocks -= 1

        if all(total_acc[b] >= n for b in range(num_blocks)):                        # :719-721
            break

    ret = final_ret()                                                                # :725-736
    fwd.trim(fwd.kv_len() - (prompt_len + len(ret)))
    return last_next_token, ret, iters


# --------------------------------------------------------------------------------------------------------------
# driver protocol (MR_humaneval.py:152-250): explicit RNG so iteration counts are reproducible
# --------------------------------------------------------------------------------------------------------------
@dataclass
class DriverResult:
    generated: List[int]
    iters: List[int]
    calls: int
    stop_reason: str
    total_new_tokens: int

    @property
    def total_iterations(self) -> int:
        return sum(self.iters)


def hf_driver(fwd, prompt: Sequence[int], n: int, max_new_tokens: int, rng, *, mode: str = "multiblock",
              K: int = 2, r: float = 0.85, lookahead_start_ratio: float = 0.0, n_gram_pool_size: int = 4,
              eos: Optional[int] = None, pad: Optional[int] = None, max_calls: int = 1024,
              max_iteration_count: int = 128, trace: Optional[Trace] = None) -> DriverResult:
    """`rng.choice(list)` supplies every random draft token (random.Random(seed) reproduces the reference's
    random.choice calls, :176-180 and :210-215).  mode = "multiblock" | "single"."""
    generated = list(prompt)
    prompt_len = len(prompt)
    iters: List[int] = []
    calls = 0
    total_new_tokens = 0
    prev_len = prompt_len
    prefill_phase = True
    first_correct = None
    prefill_drafted: List[int] = []
    stop_reason = ""
    while True:
        gen_part = generated[prompt_len:]
        if eos is not None and eos in gen_part:            # :154-161
            stop_reason = "eos"
            break
        if total_new_tokens >= max_new_tokens:             # :162-165
            stop_reason = "max_new_tokens"
            break
        if calls >= max_calls:
            stop_reason = "max_calls"
            break
        if prefill_phase:                                  # :174-198
            draft = [rng.choice(generated) for _ in range(n)]
            first_correct, prefill_drafted = hf_prefill(fwd, prompt, draft, trace)
            prefill_phase = False
            itr = 0
        else:
            if calls == 1:                                 # :206-208
                input_ids = list(prefill_drafted)
            else:                                          # :209-215
                input_ids = [first_correct] + [rng.choice(generated) for _ in range(n - 1)]
            if mode == "multiblock":
                first_correct, acc, itr = hf_multiblock(
                    fwd, input_ids, n, K=K, r=r, lookahead_start_ratio=lookahead_start_ratio,
                    n_gram_pool_size=n_gram_pool_size, eos=eos, pad=pad,
                    max_iteration_count=max_iteration_count, trace=trace)
            else:
                first_correct, acc, itr = hf_single_block(fwd, input_ids, n, eos=eos, trace=trace)
            generated = generated + list(acc)              # :232
        calls += 1
        iters.append(itr)
        added = len(generated) - prev_len
        if added > 0:
            total_new_tokens += added
        prev_len = len(generated)
    return DriverResult(generated=generated[prompt_len:], iters=iters, calls=calls, stop_reason=stop_reason,
                        total_new_tokens=total_new_tokens)


# --------------------------------------------------------------------------------------------------------------
# engine convention (inference_engine/engine/jacobi_decoding.py): fixed length L, draft[0] = cached seed
# --------------------------------------------------------------------------------------------------------------
def engine_fixed_len(forward_step: Callable[[List[int], List[int]], List[int]], token_ids: List[int],
                     prefill_draft: Optional[List[int]], L: int, max_tokens: int, max_iters: int, vocab_size: int,
                     randint: Callable[[int], List[int]], eos: Optional[int] = None):
    """_generate_single_fast (:303-445).  forward_step(token_ids, draft) returns greedy[L-1] = argmax of the logits
    verifying draft[1:], computed with draft at positions [S-1 .. S+L-2] (S = len(token_ids)); draft[0] is the last
    committed token.  `randint(k)` supplies k pad tokens (torch.randint(0, vocab) in the reference, :344, :434).
    Mutates token_ids; returns (accepted, iters, tokens_per_iteration)."""
    if L <= 1:
        return [], 0, []
    accepted: List[int] = []
    per_iter: List[int] = []
    q_draft: Optional[List[int]] = None
    eos_reached = False
    iters = 0
    while not eos_reached and len(accepted) < max_tokens and iters < max_iters:      # :326
        iters += 1
        if prefill_draft is not None and len(accepted) == 0 and q_draft is None:     # :332-347
            d = [token_ids[-1]] + list(prefill_draft[:L - 1])
            if len(d) < L:
                d = d + list(randint(L - len(d)))
            prefill_draft = None
            q_draft = d
        elif q_draft is None:                                                       # _init_draft :142-171
            q_draft = [token_ids[-1]] + list(randint(L - 1))
        else:
            q_draft[0] = token_ids[-1]                                               # :197-199
        greedy = forward_step(token_ids, q_draft)                                    # :354-357
        acc_len = _leading_matches(q_draft[1:], greedy) + 1                          # :359-362
        acc_len = max(1, min(acc_len, L))
        if eos is not None and acc_len > 1 and eos in q_draft[1:acc_len]:            # :364-369
            acc_len = 1 + q_draft[1:acc_len].index(eos) + 1
            eos_reached = True
        num_spec = acc_len - 1
        if num_spec > 0:                                                             # :376-381
            token_ids.extend(q_draft[1:acc_len])
            accepted.extend(q_draft[1:acc_len])
        if acc_len == 1:                                                             # :383-392
            nt = int(greedy[0])
            token_ids.append(nt)
            accepted.append(nt)
            num_spec = 1
            if eos is not None and nt == eos:
                eos_reached = True
        per_iter.append(num_spec)
        if eos_reached or len(accepted) >= max_tokens:                               # :411-412
            break
        d = [token_ids[-1]]                                                          # :415-436
        if acc_len < L:
            remaining = greedy[1:] if acc_len == 1 else greedy[acc_len - 1:]
            d += [int(t) for t in remaining[:L - 1]]
        else:
            d += [int(greedy[-1])]
        if len(d) < L:
            d += list(randint(L - len(d)))
        q_draft = d
    return accepted, iters, per_iter


# --------------------------------------------------------------------------------------------------------------------
# Non-greedy engine policy: JacobiDecoderNonGreedy (inference_engine/engine/jacobi_decoding_nongreedy.py)
# --------------------------------------------------------------------------------------------------------------------
def sample_not_equal(draw: Callable[[], int], avoid: int, fallback: Callable[[], int], max_tries: int = 16) -> int:
    """_sample_from_probs_not_equal (:134-153): draw from p until the sample differs from `avoid` (<= 16 tries), then the
    deterministic best alternative.  `draw()` is one torch.multinomial(probs, 1); `fallback()` the argmax of p without
    `avoid`."""
    for _ in range(max_tries):
        y = int(draw())
        if y != int(avoid):
            return y
    return int(fallback())


def engine_nongreedy(forward_step: Callable, token_ids: List[int], L: int, max_tokens: int, max_iters: int,
                     randint: Callable[[int], List[int]], uniform: Callable[[int, int], float],
                     eos: Optional[int] = None):
    """_generate_single (:385-470) with _verify_block_rejection_sampling (:300-355) inlined.

    forward_step(token_ids, draft) -> (greedy[L-1], px[L-1], residual) for the logits verifying draft[1:]:
    greedy = argmax, px[t] = softmax(logits[t] / T)[draft[t+1]] (_build_target_probs :110-123), residual(t) = a token
    drawn from softmax(logits[t] / T) conditioned on != draft[t+1] (the reference: rejection loop over torch.multinomial,
    :134-153; the device: Gumbel-max over the other tokens - the same distribution).  uniform(iteration, t) is the
    torch.rand of the accept test at position t (:322); randint(k) supplies k pad tokens (torch.randint, :227, :463).
    Mutates token_ids; returns (accepted, iters, tokens_per_iteration, drafts)."""
    if L <= 1:
        return [], 0, [], []
    accepted: List[int] = []
    per_iter: List[int] = []
    drafts: List[List[int]] = []
    q_draft: Optional[List[int]] = None
    eos_reached = False
    iters = 0
    while not eos_reached and len(accepted) < max_tokens and iters < max_iters:      # :399
        iters += 1
        if q_draft is None:                                                          # _init_draft :216-236
            q_draft = [token_ids[-1]] + list(randint(L - 1))
        else:
            q_draft[0] = token_ids[-1]                                               # _resize_or_init_draft :249-250
        drafts.append(list(q_draft))
        greedy, px, residual = forward_step(token_ids, q_draft)
        committed: List[int] = []
        for t in range(L - 1):                                                       # :316-347
            proposed = int(q_draft[t + 1])
            if uniform(iters - 1, t) < float(px[t]):
                committed.append(proposed)
                if eos is not None and proposed == eos:
                    eos_reached = True
                    break
                continue
            bonus = int(residual(t))
            committed.append(bonus)
            if eos is not None and bonus == eos:
                eos_reached = True
            break
        token_ids.extend(committed)                                                  # :419-423
        accepted.extend(committed)
        per_iter.append(len(committed))
        if eos_reached or len(accepted) >= max_tokens:                               # :441-442
            break
        acc_len = 1 + len(committed)                                                 # :446-466
        d = [token_ids[-1]]
        if acc_len < L:
            remaining = greedy[acc_len - 1:] if acc_len > 1 else greedy[1:]
            d += [int(t) for t in remaining[:L - 1]]
        else:
            d += [int(greedy[-1])]
        if len(d) < L:
            d += list(randint(L - len(d)))
        q_draft = d
    return accepted, iters, per_iter, drafts


# ---- the counter-based generator of the device path (csrc/jf_policy.h philox4x32_10), restated for the parity tests ---
def philox4x32_10(c0: int, c1: int, c2: int, c3: int, k0: int, k1: int):
    M = 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        c0, c1, c2, c3 = ((p1 >> 32) ^ c1 ^ k0) & M, p1 & M, ((p0 >> 32) ^ c3 ^ k1) & M, p0 & M
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


RNG_GUMBEL, RNG_ACCEPT = 1, 2


def device_accept_uniform(seed: int, rng_offset: int, row: int, fwd: int) -> float:
    """csrc/jf_policy.h ng_accept_uniform: 24-bit uniform in [0, 1) of in-flight row `row` of forward `fwd`."""
    x = philox4x32_10(row, 0, (fwd + rng_offset) & 0xFFFFFFFF, RNG_ACCEPT, seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF)[0]
    return (x >> 8) / 16777216.0


def device_gumbel_uniforms(seed: int, rng_offset: int, row: int, fwd: int, vocab: int):
    """The (0, 1) uniforms behind the Gumbel noise of in-flight row `row` over the whole vocabulary, as a numpy fp32
    array (csrc/jf_gemm.cuh EPI_SAMPLE: counter = (token, row >> 2, forward, RNG_GUMBEL), word row & 3)."""
    import numpy as np
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    c0 = np.arange(vocab, dtype=np.uint64)
    c1 = np.full(vocab, row >> 2, dtype=np.uint64)
    c2 = np.full(vocab, (fwd + rng_offset) & 0xFFFFFFFF, dtype=np.uint64)
    c3 = np.full(vocab, RNG_GUMBEL, dtype=np.uint64)
    M = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        n0 = ((p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0)) & M
        n1 = p1 & M
        n2 = ((p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1)) & M
        n3 = p0 & M
        c0, c1, c2, c3 = n0, n1, n2, n3
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    word = (c0, c1, c2, c3)[row & 3]
    return (((word >> np.uint64(8)).astype(np.float32) + np.float32(0.5)) * np.float32(1.0 / 16777216.0)).astype(np.float32)
