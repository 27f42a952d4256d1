"""The barrier protocols of the tcgen05 kernels, restated as little programs and explored over EVERY interleaving,
without a GPU.  First and in most detail the prefill attention kernel (hymt2sharp_b200/csrc/attention_prefill_tc.cu);
the decode attention and the matrix products follow at the end.

Why: a wait on an mbarrier names a parity, and a parity cannot tell a phase from the one two later.  A reader that
falls two phases behind its barrier waits for ever; one that is a phase early passes at once.  Whether that can
happen does not depend on likelihoods (a thread may be kept from running for any length of time) but on who has to
wait for whom, and that can be enumerated.  The roles, as in the kernel:

  producer       Q with K(0); then for every tile i: wait "stage i mod 2 free" (tile i - 2), copy K(i + 1) with V(i)
  score issuer   S(0); then for i: wait copy i, release its hold on the stage, wait P·V(i - 2), wait P(i - 1), issue S(i + 1)
  P·V issuer     for i: wait P(i), wait copy i, issue P·V(i), whose completion frees the stage and completes O's barrier
  softmax        for i: wait S(i), sometimes wait P·V(i - 1) (a maximum rose), on the last tile sometimes wait copy i,
                 announce P(i); at the end wait P·V of the last tile

Copies land and products complete at any later time (products of one issuer in order).  A first version with two
barriers for P, two for O and the stage held by P·V alone met the never-ending wait on the device; the exploration
finds it in that version within milliseconds, and finds none in the kernel's.

The numbers that the little programs are built from (stages, K slots, barriers per purpose, holders of a stage,
accumulators, issuers) are not written here: they come out of the compiled kernels (ops.protocol_numbers, which
returns the .cu files' own constants), so a change of one of them in a kernel changes what is explored."""
import pytest

from hymt2sharp_b200.kernels import ops

NUMBERS = ops.protocol_numbers()


def explore(roles, sizes, arrivals_needed=None):
    """roles: programs of ("wait" | "wait or not", barrier, index, phase), ("arrive", barrier, index),
    ("copy", barrier, index) — lands at any later time — and ("issue", queue, [(barrier, index), ...]) — completes at
    any later time after the products issued before it on the same queue, and then arrives at its barriers.  ("must", barrier, index,
    phase) is no wait: going on while that phase is not complete is what goes wrong (memory that others have yet to read is written).
    sizes: barriers of each name; arrivals_needed: arrivals that complete a phase (1 unless named).
    Returns None when no interleaving goes wrong, else a sentence about the first one found that does."""
    arrivals_needed = arrivals_needed or {}
    at, total = {}, 0
    for name, n in sizes.items():
        at[name] = total
        total += n
    queues = sorted({op[1] for role in roles for op in role if op[0] == "issue"})

    def arrive(done, held, bar, idx):
        done, held = list(done), list(held)
        held[at[bar] + idx] += 1
        if held[at[bar] + idx] == arrivals_needed.get(bar, 1):
            held[at[bar] + idx] = 0
            done[at[bar] + idx] += 1
        return tuple(done), tuple(held)

    # (each role's place, completed phases of every barrier, arrivals at the open phases, copies in flight, products in flight)
    first = ((0,) * len(roles), (0,) * total, (0,) * total, (), tuple(() for _ in queues))
    seen, todo = {first}, [first]
    while todo:
        places, done, held, copies, issued = todo.pop()
        after = []
        for r, role in enumerate(roles):
            if places[r] >= len(role):
                continue
            op = role[places[r]]
            moved = places[:r] + (places[r] + 1,) + places[r + 1:]
            if op[0] in ("wait", "wait or not"):
                _, bar, idx, phase = op
                complete = done[at[bar] + idx]
                if op[0] == "wait or not":
                    after.append((moved, done, held, copies, issued))
                if (complete & 1) != (phase & 1):      # what the parity test sees
                    if complete != phase + 1:
                        return f"role {r} passes its wait for phase {phase} of {bar}[{idx}] with {complete} phases complete"
                    after.append((moved, done, held, copies, issued))
            elif op[0] == "must":
                _, bar, idx, phase = op
                if done[at[bar] + idx] <= phase:
                    return f"role {r} goes on without phase {phase} of {bar}[{idx}]"
                after.append((moved, done, held, copies, issued))
            elif op[0] == "arrive":
                d, h = arrive(done, held, op[1], op[2])
                after.append((moved, d, h, copies, issued))
            elif op[0] == "copy":
                after.append((moved, done, held, tuple(sorted(copies + ((op[1], op[2]),))), issued))
            else:
                q = queues.index(op[1])
                after.append((moved, done, held, copies, issued[:q] + (issued[q] + (tuple(op[2]),),) + issued[q + 1:]))
        for j, (bar, idx) in enumerate(copies):            # a copy lands
            d, h = arrive(done, held, bar, idx)
            after.append((places, d, h, copies[:j] + copies[j + 1:], issued))
        for q in range(len(queues)):                       # the oldest product of a queue is complete
            if issued[q]:
                d, h = done, held
                for bar, idx in issued[q][0]:
                    d, h = arrive(d, h, bar, idx)
                after.append((places, d, h, copies, issued[:q] + (issued[q][1:],) + issued[q + 1:]))
        if not after and any(places[r] < len(role) for r, role in enumerate(roles)):
            stuck = [role[places[r]] for r, role in enumerate(roles) if places[r] < len(role)]
            return f"nothing can move any more: {stuck}"
        for state in after:
            if state not in seen:
                seen.add(state)
                todo.append(state)
    return None


def prefill(tiles, p_bars, o_bars, stage_holders, kv_stages=None):
    kv = kv_stages or NUMBERS["prefill"]["kv_stages"]
    assert NUMBERS["prefill"]["s_buffers"] == 2     # the score buffers go by a tile's parity, here as in the kernel
    producer = [("copy", "q", 0)]
    for i in range(tiles):
        if i >= kv:
            producer.append(("wait", "stage_free", i % kv, i // kv - 1))
        producer.append(("copy", "copied", i % kv))
    scores = [("wait", "q", 0, 0), ("issue", "S", [("s_done", 0)])]
    for i in range(tiles - 1):
        scores.append(("wait", "copied", i % kv, i // kv))
        if stage_holders == 2:
            scores.append(("arrive", "stage_free", i % kv))
        if i >= 2:
            scores.append(("wait", "o_done", (i - 2) % o_bars, (i - 2) // o_bars))
        if i >= 1:
            scores.append(("wait", "p_written", (i - 1) % p_bars, (i - 1) // p_bars))
        scores.append(("issue", "S", [("s_done", (i + 1) & 1)]))
    weighted = []
    for i in range(tiles):
        weighted.append(("wait", "p_written", i % p_bars, i // p_bars))
        weighted.append(("wait", "copied", i % kv, i // kv))
        weighted.append(("issue", "PV", [("stage_free", i % kv), ("o_done", i % o_bars)]))
    softmax = []
    for i in range(tiles):
        softmax.append(("wait", "s_done", i & 1, i >> 1))
        if i > 0:
            softmax.append(("wait or not", "o_done", (i - 1) % o_bars, (i - 1) // o_bars))
        if i == tiles - 1:
            softmax.append(("wait or not", "copied", i % kv, i // kv))
        softmax.append(("arrive", "p_written", i % p_bars))
    softmax.append(("wait", "o_done", (tiles - 1) % o_bars, (tiles - 1) // o_bars))
    sizes = {"q": 1, "copied": kv, "stage_free": kv, "s_done": 2, "o_done": o_bars, "p_written": p_bars}
    return explore((producer, scores, weighted, softmax), sizes, {"stage_free": stage_holders})


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 8, 13, 32])
def test_no_interleaving_of_the_kernels_protocol_goes_wrong(tiles):
    n = NUMBERS["prefill"]     # as compiled: 2 stages, 3 barriers for P (one per K slot), 3 for O, 2 holders of a stage
    assert n["p_bars"] == n["k_slots"]
    assert prefill(tiles, p_bars=n["p_bars"], o_bars=n["o_bars"], stage_holders=n["stage_holders"]) is None


@pytest.mark.parametrize("p_bars, o_bars, stage_holders", [(2, 2, 1), (2, 3, 2), (3, 2, 2), (3, 3, 1)])
def test_each_of_the_three_measures_is_needed(p_bars, o_bars, stage_holders):
    """Two barriers for P (the version that hung on the device), two for O, or a stage that only P·V holds: each
    has an interleaving in which a reader is two phases behind and nothing can move any more."""
    found = [prefill(tiles, p_bars, o_bars, stage_holders) for tiles in (3, 4, 5, 6)]
    assert any(found), found


# ---- the decode attention kernel (hymt2sharp_b200/csrc/attention_decode_tc.cu), one round of a CTA's items ----
#   producer       the first three items' copies at once; then for item n: wait "stage n mod 3 free" (item n - 3), copy K with Q, copy V
#   score issuer   for n: wait K and Q of n, wait "accumulators n mod 2 free" (item n - 2), issue S(n)
#   P·V issuer     for n: wait P(n), wait V(n), issue P·V(n), whose completion completes O's barrier and frees the stage;
#                  at the end it waits for the last stages to be free
#   softmax groups group g takes the items n = g, g + 2, ...: wait S(n), sometimes wait V(n) (rows to clear), announce P(n),
#                  wait O(n), free the accumulators
def decode(items):
    stages = NUMBERS["decode"]["stages"]
    assert NUMBERS["decode"]["accumulators"] == 2   # two groups of softmax warps take turns, here as in the kernel
    producer, scores, weighted, groups = [], [], [], ([], [])
    for n in range(items):
        s, t = n % stages, n & 1
        if n >= stages:
            producer.append(("wait", "stage_free", s, n // stages - 1))
        producer += [("copy", "kq_full", s), ("copy", "v_full", s)]
        scores.append(("wait", "kq_full", s, n // stages))
        if n >= 2:
            scores.append(("wait", "tmem_free", t, (n >> 1) - 1))
        scores.append(("issue", "S", [("s_done", t)]))
        weighted += [("wait", "p_ready", t, n >> 1), ("wait", "v_full", s, n // stages),
                     ("issue", "PV", [("o_done", t), ("stage_free", s)])]
        groups[t].extend([("wait", "s_done", t, n >> 1), ("wait or not", "v_full", s, n // stages), ("arrive", "p_ready", t),
                          ("wait", "o_done", t, n >> 1), ("arrive", "tmem_free", t)])
    for m in range(max(0, items - stages), items):
        weighted.append(("wait", "stage_free", m % stages, m // stages))
    sizes = {"kq_full": stages, "v_full": stages, "stage_free": stages, "s_done": 2, "p_ready": 2, "o_done": 2, "tmem_free": 2}
    return explore((producer, scores, weighted, groups[0], groups[1]), sizes)


@pytest.mark.parametrize("items", [1, 2, 3, 4, 7, 12])
def test_no_interleaving_of_the_decode_attentions_protocol_goes_wrong(items):
    assert decode(items) is None


# ---- the persistent matrix product (hymt2sharp_b200/csrc/gemm_tc.cu): a ring of stages across tiles, two accumulators ----
#   producer   for every k block: wait "stage free" (the block a ring earlier), copy the stage
#   issuer     for every tile j: wait "accumulator j mod 2 drained" (tile j - 2); for its k blocks: wait the stage, issue the
#              MMAs (their completion frees the stage); then the tile's completion fills the accumulator's barrier
#   epilogue   group g, for the tiles g, g + groups, ...: wait the accumulator, drain it, announce it empty; then help with
#              the last tile if it is the other group's
# (the looks ahead at the next stage's barrier are reads of the same reader in the same order: nothing new for this model)
def persistent_gemm(tiles, k_blocks, stages, groups=None):
    groups = groups or NUMBERS["gemm"]["epilogue_groups"]
    producer, issuer, epilogues = [], [], [[] for _ in range(groups)]
    block = 0
    for j in range(tiles):
        if j >= 2:
            issuer.append(("wait", "acc_empty", j & 1, (j >> 1) - 1))
        for _ in range(k_blocks):
            s, use = block % stages, block // stages
            if use > 0:
                producer.append(("wait", "empty", s, use - 1))
            producer.append(("copy", "full", s))
            issuer += [("wait", "full", s, use), ("issue", "MMA", [("empty", s)])]
            block += 1
        issuer.append(("issue", "MMA", [("acc_full", j & 1)]))
        epilogues[j % groups] += [("wait", "acc_full", j & 1, j >> 1), ("arrive", "acc_empty", j & 1)]
    if groups == 2:
        # the CTA's last tile is drained by both groups: the group that does not own it waits for its accumulator too,
        # on a barrier whose earlier phases it has not followed, once it is through with its own tiles
        last = tiles - 1
        epilogues[1 - last % 2].append(("wait", "acc_full", last & 1, last >> 1))
    return explore((producer, issuer, *epilogues), {"full": stages, "empty": stages, "acc_full": 2, "acc_empty": 2})


@pytest.mark.parametrize("tiles, k_blocks, stages", [(1, 1, 4), (3, 2, 4), (5, 3, 2), (6, 4, 5), (4, 9, 4),
                                                     (3, 10, NUMBERS["gemm"]["max_stages"])])
def test_no_interleaving_of_the_persistent_products_protocol_goes_wrong(tiles, k_blocks, stages):
    assert NUMBERS["gemm"]["accumulators"] == 2 and 2 <= stages <= NUMBERS["gemm"]["max_stages"]
    assert NUMBERS["gemm"]["epilogue_groups"] in (1, 2)   # a group per accumulator, or one group for both
    assert persistent_gemm(tiles, k_blocks, stages) is None
    assert persistent_gemm(tiles, k_blocks, stages, groups=1) is None


# ---- the same by pairs of CTAs: the even one's issuer and barriers for what both bring, both CTAs' for what they are given back ----
#   producer r     its rows of both operands, counted at the even CTA's stage (which the even producer arms: one arrival more)
#   issuer (even)  as above; its completions free the stage in both CTAs and fill the accumulator's barrier in both
#   epilogue r     drains its CTA's half and announces that at the even CTA (`acc_empty` wants both)
def pair_gemm(tiles, k_blocks, stages, groups=None):
    groups = groups or NUMBERS["gemm"]["epilogue_groups"]
    producers, issuer, epilogues = ([], []), [], [[] for _ in range(2 * groups)]
    block = 0
    for j in range(tiles):
        if j >= 2:
            issuer.append(("wait", "acc_empty", j & 1, (j >> 1) - 1))
        for _ in range(k_blocks):
            s, use = block % stages, block // stages
            for r, producer in enumerate(producers):
                if use > 0:
                    producer.append(("wait", f"empty{r}", s, use - 1))
                producer += ([("arrive", "full", s)] if r == 0 else []) + [("copy", "full", s)]
            issuer += [("wait", "full", s, use), ("issue", "MMA", [("empty0", s), ("empty1", s)])]
            block += 1
        issuer.append(("issue", "MMA", [("acc_full0", j & 1), ("acc_full1", j & 1)]))
        for r in range(2):
            epilogues[r * groups + j % groups] += [("wait", f"acc_full{r}", j & 1, j >> 1), ("arrive", "acc_empty", j & 1)]
    if groups == 2:
        last = tiles - 1
        for r in range(2):
            epilogues[r * groups + 1 - last % 2].append(("wait", f"acc_full{r}", last & 1, last >> 1))
    sizes = {"full": stages, "empty0": stages, "empty1": stages, "acc_full0": 2, "acc_full1": 2, "acc_empty": 2}
    return explore((*producers, issuer, *epilogues), sizes, {"full": 3, "acc_empty": 2})


@pytest.mark.parametrize("tiles, k_blocks, stages", [(1, 1, 4), (3, 2, 4), (5, 3, 2), (4, 4, 3)])
def test_no_interleaving_of_the_pairs_protocol_goes_wrong(tiles, k_blocks, stages):
    assert pair_gemm(tiles, k_blocks, stages) is None
    assert pair_gemm(tiles, k_blocks, stages, groups=1) is None


# ---- the tile kernel of the matrix product with several MMA issuers (few tokens): who may read which stage's barrier ----
#   producer   for every k block i: wait "stage i mod stages free" (block i - stages), copy the stage
#   issuer j   takes some of the k blocks: wait the stage, issue its MMAs into an accumulator of its own (they free the stage)
# "own": issuer j takes the blocks that land in the stages j, j + issuers, ... (what the kernel does); otherwise the blocks
# j, j + issuers, ... round-robin, which was the first version: an issuer then met a stage's barrier only every few phases.
def tile_gemm(blocks, stages, issuers, own):
    producer = []
    takers = [[] for _ in range(issuers)]
    for i in range(blocks):
        s = i % stages
        if i >= stages:
            producer.append(("wait", "empty", s, i // stages - 1))
        producer.append(("copy", "full", s))
        j = s % issuers if own else i % issuers
        takers[j] += [("wait", "full", s, i // stages), ("issue", f"MMA{j}", [("empty", s)])]
    return explore((producer, *takers), {"full": stages, "empty": stages})


@pytest.mark.parametrize("blocks, stages", [(32, 5), (12, 6), (20, 3), (7, 2), (18, 4), (40, NUMBERS["gemm"]["max_stages"])])
@pytest.mark.parametrize("issuers", sorted({1, NUMBERS["gemm"]["issuers"]}))
def test_issuers_that_own_their_stages_never_misread_a_barrier(blocks, stages, issuers):
    assert NUMBERS["gemm"]["issuers_own_stages"] == 1
    assert tile_gemm(blocks, stages, issuers, own=True) is None


def test_three_issuers_taking_turns_over_five_stages_did():
    """The version that ended two launches with a fault: an issuer took a stage whose copy had not landed."""
    assert "passes its wait" in tile_gemm(32, 5, 3, own=False)


# ---- the float32 product (hymt2sharp_b200/csrc/gemm_f32_tc.cu): stages of W are cut into pieces, two stages a chunk ----
#   producer        for every stage i: wait "stage free" (the stage a ring earlier), copy the stage
#   converter g     for the stages i = g, g + groups, ...: wait the stage, wait "buffer free" (the chunk `buffers` earlier is
#                   multiplied), free the stage, announce half of chunk i div 2 (two arrivals complete it)
#   planes          (where the tokens' pieces come ready) for every chunk j: wait "slot free", copy the slot
#   issuer g of 2   for the chunks j = g, g + 2, ...: wait its accumulator drained (chunk j - 2) and the pieces of chunk j, in that
#                   order; issue its MMAs, which free the buffer (and the slot) and complete the chunk
#   drain           for every chunk: wait it complete, announce its accumulator drained
# (where two barriers are looked at behind one another first, that is these waits passing without delay)
def f32_product(chunks, groups, buffers, stages, slots=0, drained_first=True):
    producer, drain, planes = [], [], []
    converters, issuers = [[] for _ in range(groups)], ([], [])
    for i in range(2 * chunks):
        s, buf, use = i % stages, i // 2 % buffers, i // 2 // buffers
        if i >= stages:
            producer.append(("wait", "empty", s, i // stages - 1))
        producer.append(("copy", "full", s))
        freed = [("wait", "freed", buf, use - 1)] if use else []
        converters[i % groups] += [("wait", "full", s, i // stages), *freed, ("arrive", "empty", s), ("arrive", "ready", buf)]
    for j in range(chunks):
        buf, g, use = j % buffers, j % 2, j // 2
        drained = [("wait", "drained", g, use - 1)] if use else []
        ready = [("wait", "ready", buf, j // buffers)]
        frees = [("freed", buf), ("done", g)]
        if slots:
            planes += [("wait", "slot_free", j % slots, j // slots - 1)] if j >= slots else []
            planes.append(("copy", "slot_full", j % slots))
            issuers[g].append(("wait", "slot_full", j % slots, j // slots))
            frees = [("slot_free", j % slots)] + frees
        issuers[g].extend((drained + ready if drained_first else ready + drained) + [("issue", f"MMA{g}", frees)])
        drain += [("wait", "done", g, use), ("arrive", "drained", g)]
    sizes = dict(full=stages, empty=stages, ready=buffers, freed=buffers, done=2, drained=2, slot_full=max(slots, 1), slot_free=max(slots, 1))
    return explore((producer, *converters, *issuers, drain, planes), sizes, {"ready": 2})


@pytest.mark.parametrize("rows, chunks", [(16, 1), (16, 9), (32, 7), (64, 1), (64, 4), (64, 7), (64, 10)])
def test_no_interleaving_of_the_float32_products_protocol_goes_wrong(rows, chunks):
    n, form = NUMBERS["f32"], "few" if rows <= 32 else "wide"
    planes, _, stages, _, _ = ops.gemm_f32_tc_plan(rows, 2048, 64 * chunks)
    assert not planes and n["drained_first"] == 1
    assert f32_product(chunks, n[form + "_groups"], n[form + "_buffers"], stages) is None


@pytest.mark.parametrize("chunks, stages", [(1, 4), (4, 4), (3, 6)])
def test_no_interleaving_of_the_float32_products_protocol_with_planes_goes_wrong(chunks, stages):
    n = NUMBERS["f32"]
    assert f32_product(chunks, n["planes_groups"], n["planes_buffers"], stages, n["plane_slots"]) is None
    assert f32_product(chunks + 2, n["planes_groups"], n["planes_buffers"], stages, 2) is None      # (fewer slots: more reuse in fewer chunks)


def test_the_float32_products_two_rules_are_needed():
    """Pieces looked at before the accumulator is drained (tiles of 64 rows did, three buffers between two issuers): the parity of the phase before the
    last passes.  Four groups of converters over eight stages instead of four: so does a buffer's, in front of the writes."""
    n = NUMBERS["f32"]
    assert "of ready" in f32_product(4, n["wide_groups"], n["wide_buffers"], 4, drained_first=False)
    assert f32_product(4, n["wide_groups"], n["wide_buffers"], 4) is None
    for rows in (33, 64):
        assert ops.gemm_f32_tc_plan(rows, 2048, 2048)[2] == 4


# ---- the grouped product of few rows (hymt2sharp_b200/csrc/gemm_grouped_few.cu): a CTA by itself, then what a cluster's CTAs hand each other ----
#   producer   for every weight block: wait "stage free", copy it
#   loaders    for the q-th row tile of the CTA's items: wait "rows free" (tile q - 2), announce the rows (all loaders)
#   issuer     an item of another row tile: wait its rows; for every block: wait the stage, wait "accumulator drained" (`accs` blocks
#              earlier), issue (frees the stage, completes the accumulator); behind a row tile's last item a completion frees its rows
#   sums       for every block: wait the accumulator, announce it drained
def few_rows_cta(items, blocks, stages, accs, loaders):
    producer, rows, issuer, sums = [], [], [], []
    q, tile, j = -1, None, 0
    for n, item in enumerate(items):
        if item != tile:
            tile, q = item, q + 1
            if q >= 2:
                rows.append(("wait", "rows_free", q & 1, (q >> 1) - 1))
            rows.append(("arrive", "rows_full", q & 1))
            issuer.append(("wait", "rows_full", q & 1, q >> 1))
        for _ in range(blocks):
            s, use = j % stages, j // stages
            if use > 0:
                producer.append(("wait", "empty", s, use - 1))
            producer.append(("copy", "full", s))
            issuer.append(("wait", "full", s, use))
            if j >= accs:
                issuer.append(("wait", "acc_empty", j % accs, j // accs - 1))
            issuer.append(("issue", "MMA", [("empty", s), ("acc_full", j % accs)]))
            sums += [("wait", "acc_full", j % accs, j // accs), ("arrive", "acc_empty", j % accs)]
            j += 1
        if n + 1 < len(items) and items[n + 1] != tile:
            issuer.append(("issue", "MMA", [("rows_free", q & 1)]))
    sizes = {"full": stages, "empty": stages, "acc_full": accs, "acc_empty": accs, "rows_full": 2, "rows_free": 2}
    return explore((producer, *[rows] * loaders, issuer, sums), sizes, {"rows_full": loaders})


@pytest.mark.parametrize("items, blocks, stages", [([0], 1, 2), ([0, 0, 0], 2, 2), ([0, 1, 2, 3, 4], 1, 2), ([0, 0, 1, 2, 2, 3], 2, 3), ([3, 4, 4, 4, 5, 6], 1, 8)])
def test_no_interleaving_of_the_few_rows_protocol_within_a_cta_goes_wrong(items, blocks, stages):
    n = NUMBERS["grouped_few"]
    assert n["max_inner"] == ops.FEW_MAX_INNER and n["row_buffers"] == 2 and 2 <= stages <= n["max_stages"]
    assert few_rows_cta(items, blocks, stages, n["accumulators"], n["loader_warps"]) is None


def few_rows_cluster(items, ranks, warps, buffers):
    """Every summing warp of every CTA, item after item: write its sums into each CTA's buffer, announce them there, wait for all of them in its own CTA,
    read.  Writing while a warp of the CTA written to has yet to read what stood in that buffer is what must not happen."""
    roles = []
    for r in range(ranks):
        for _ in range(warps):
            role = []
            for n in range(items):
                b, use = n % buffers, n // buffers
                if use > 0:
                    role += [("must", f"read{q}", b, use - 1) for q in range(ranks)]
                role += [("arrive", f"parts{q}", b) for q in range(ranks)]
                role += [("wait", f"parts{r}", b, use), ("arrive", f"read{r}", b)]
            roles.append(role)
    sizes = {f"{kind}{q}": buffers for kind in ("parts", "read") for q in range(ranks)}
    return explore(tuple(roles), sizes, {**{f"parts{q}": ranks * warps for q in range(ranks)}, **{f"read{q}": warps for q in range(ranks)}})


@pytest.mark.parametrize("items, ranks, warps", [(1, 4, 1), (4, 2, 2), (5, 3, 1), (7, 2, 1)])
def test_no_interleaving_of_the_few_rows_protocol_between_ctas_goes_wrong(items, ranks, warps):
    assert NUMBERS["grouped_few"]["ranks"] >= ranks
    assert few_rows_cluster(items, ranks, warps, NUMBERS["grouped_few"]["sum_buffers"]) is None


def test_the_few_rows_sums_need_two_buffers():
    assert "goes on without" in few_rows_cluster(3, 2, 1, 1)


def gated_drain(tiles, gives_up, walks_on):
    """The warps of a gated drain group, which meet twice a tile at a barrier that has no limit.  gives_up[w]: the tile in which warp w's bounded wait
    gives up (None: never); with `walks_on` it meets the others in that tile and all that follow."""
    roles = []
    for mine in gives_up:
        meets = 2 * (tiles if mine is None or walks_on else mine)
        roles.append([op for phase in range(meets) for op in (("arrive", "meet", 0), ("wait", "meet", 0, phase))])
    return explore(tuple(roles), {"meet": 1}, {"meet": len(gives_up)})


@pytest.mark.parametrize("gives_up", [(None, None, None, None), (0, None, None, None), (None, 2, None, None), (1, 1, None, 2), (2, 2, 2, 2), (0, 1, 2, None)])
def test_a_warp_that_gives_up_still_meets_its_gated_drain_group(gives_up):
    n = NUMBERS["f32"]
    assert n["gated_walks_on"] == 1 and n["gated_warps"] == len(gives_up)
    assert gated_drain(3, gives_up, walks_on=True) is None
    if len(set(gives_up)) > 1:      # leaving, as it did: the others stand at the barrier for ever
        assert "nothing can move" in gated_drain(3, gives_up, walks_on=False)
