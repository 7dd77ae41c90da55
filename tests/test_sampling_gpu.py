"""Temperature / top-k sampling kernel (q3_sample through the C ABI) against the rule stated in PyTorch fp64.

The kernel works in fp32, so a row whose uniform number falls within 1e-4 of a boundary of the exact cumulative
distribution may land on either side: the gate is that the chosen token's CDF interval, widened by that much,
contains u, that the token belongs to the kept set, and that many draws reproduce the exact probabilities."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

CDF_TOL = 1e-4


def exact(logits, temperature, top_k):
    rows = logits.double().cpu()
    keep = torch.ones_like(rows, dtype=torch.bool)
    if 0 < top_k < rows.shape[-1]:
        keep = rows >= rows.topk(top_k, dim=-1).values[:, -1:]
    w = torch.where(keep, torch.exp((rows - rows.max(dim=-1, keepdim=True).values) / temperature), torch.zeros_like(rows))
    return keep, w / w.sum(dim=-1, keepdim=True)


@pytest.mark.parametrize("vocab,batch", [(151936, 4), (4096, 33), (1000, 7), (17, 3)])
@pytest.mark.parametrize("temperature,top_k", [(1.0, 0), (0.7, 50), (1.5, 5), (0.3, 1000), (1.0, 2)])
def test_sampled_token_matches_the_exact_distribution_function(vocab, batch, temperature, top_k):
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(vocab + batch + top_k)
    logits = (torch.randn(batch, vocab, generator=g) * 3.0).cuda()
    u = torch.rand(batch, generator=g).cuda()
    got = sampling.sample(logits, temperature, top_k, u=u).cpu()
    keep, prob = exact(logits, temperature, top_k)
    cdf = prob.cumsum(dim=-1)
    for b in range(batch):
        j = int(got[b])
        assert 0 <= j < vocab and bool(keep[b, j]), f"row {b}: token {j} is outside the kept set"
        lo = float(cdf[b, j - 1]) if j else 0.0
        assert lo - CDF_TOL <= float(u[b]) <= float(cdf[b, j]) + CDF_TOL, f"row {b}: u {float(u[b]):.6f} outside [{lo:.6f}, {float(cdf[b, j]):.6f}]"
    # the stated rule in PyTorch agrees wherever u is not within the tolerance of a boundary
    ref = sampling.sample_reference(logits, temperature, top_k, u).cpu()
    for b in range(batch):
        if int(ref[b]) != int(got[b]):
            edge = torch.cat([torch.zeros(1, dtype=torch.float64), cdf[b]])
            assert float((edge - float(u[b])).abs().min()) <= CDF_TOL, f"row {b}: kernel {int(got[b])}, rule {int(ref[b])}"


def test_argmax_cases_and_ties():
    from qwen3mk import sampling

    logits = torch.zeros(3, 2048)
    logits[0, 77] = 5.0
    logits[1, [9, 1200]] = 4.0           # a tie: the lowest index wins
    logits[2] = -1.0
    logits = logits.cuda()
    assert sampling.sample(logits, 0.0, 0).tolist() == [77, 9, 0]
    assert sampling.sample(logits, 1.0, 1).tolist() == [77, 9, 0]
    # ties at the k-th value are all kept: with k = 1 + ... the two tied logits share the mass
    u = torch.tensor([0.1, 0.9, 0.5]).cuda()
    got = sampling.sample(logits, 1.0, 2, u=u).tolist()
    assert got[1] in (9, 1200) and got[0] in range(2048)


def test_many_draws_follow_the_probabilities():
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(5)
    base = torch.randn(50, generator=g) * 2.0
    n = 20000
    logits = base.repeat(n, 1).cuda()
    toks = sampling.sample(logits, 0.8, 10, generator=torch.Generator(device="cuda").manual_seed(1)).cpu()
    _, prob = exact(base[None], 0.8, 10)
    freq = torch.bincount(toks, minlength=50).double() / n
    assert float((freq - prob[0]).abs().max()) < 0.015
    assert float(freq[prob[0] == 0].sum()) == 0.0


def test_sampled_stream_feeds_the_next_launch(oracle):
    """The sampled token is written into the token buffer the next launch reads: no host round trip."""
    from qwen3mk import Megakernel, sampling

    shp = oracle.Shape(layers=2, vocab=4096)
    inp = oracle.synthetic(3, shp, context=30)
    dev = {k: v.cuda() for k, v in inp.items()}
    mk = Megakernel(layers=2, vocab=4096)
    out = mk.bind(dev, grow=8)                       # unchained: every launch reads dev["token"]
    gen = torch.Generator(device="cuda").manual_seed(0)
    toks = []
    for _ in range(8):
        mk.launch()
        sampling.sample(out["logits"], 0.9, 40, generator=gen, out=dev["token"])
        toks.append(dev["token"].clone())
    mk.status()
    toks = torch.stack(toks).cpu().tolist()
    assert all(0 <= t < 4096 for t in toks)
    # the same seed reproduces the stream
    dev2 = {k: v.cuda() for k, v in inp.items()}
    mk2 = Megakernel(layers=2, vocab=4096)
    out2 = mk2.bind(dev2, grow=8)
    gen = torch.Generator(device="cuda").manual_seed(0)
    toks2 = []
    for _ in range(8):
        mk2.launch()
        sampling.sample(out2["logits"], 0.9, 40, generator=gen, out=dev2["token"])
        toks2.append(int(dev2["token"]))
    assert toks2 == toks


@pytest.mark.parametrize("vocab,batch", [(1, 2), (31, 1), (2047, 3), (2049, 1), (32768, 1), (32769, 9), (151936, 17), (151937, 65)])
@pytest.mark.parametrize("top_k", [0, 2, 64, 5000])
def test_every_split_of_a_row_over_blocks(vocab, batch, top_k):
    """Rows on 1, 2, 4, 8 and 16 blocks, elements in registers or re-read, runs that end inside a block: fp64 rule, as above."""
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(vocab * 7 + batch + top_k)
    logits = torch.randn(batch, vocab, generator=g) * 3.0
    logits[0, vocab // 2:] = float("-inf") if vocab > 1 else 0.0      # half the words of a row masked out
    u = torch.rand(batch, generator=g)
    got = sampling.sample(logits.cuda(), 0.9, top_k, u=u.cuda()).cpu()
    keep, prob = exact(logits, 0.9, top_k)
    cdf = prob.cumsum(dim=-1)
    for b in range(batch):
        j = int(got[b])
        assert 0 <= j < vocab and bool(keep[b, j])
        lo = float(cdf[b, j - 1]) if j else 0.0
        assert lo - CDF_TOL <= float(u[b]) <= float(cdf[b, j]) + CDF_TOL
    assert sampling.sample(logits.cuda(), 0.0, 0).cpu().tolist() == logits.argmax(dim=-1).tolist()


@pytest.mark.parametrize("top_k", [3, 700, 9000])
def test_thousands_of_equal_logits_at_the_threshold_are_all_kept(top_k):
    """More candidates than a block publishes: the radix select decides.  Two larger words and 10000 equal ones."""
    from qwen3mk import sampling

    vocab = 40000
    logits = torch.full((1, vocab), -4.0)
    logits[0, 5000:15000] = 1.0
    logits[0, [123, 39999]] = 2.0
    keep, prob = exact(logits, 1.0, top_k)
    assert int(keep.sum()) == 10002
    cdf = prob.cumsum(dim=-1)[0]
    u = torch.linspace(0.001, 0.999, 50)
    got = sampling.sample(logits.repeat(50, 1).cuda(), 1.0, top_k, u=u.cuda()).cpu()
    for b in range(50):
        j = int(got[b])
        assert bool(keep[0, j])
        assert (float(cdf[j - 1]) if j else 0.0) - CDF_TOL <= float(u[b]) <= float(cdf[j]) + CDF_TOL


@pytest.mark.parametrize("vocab", [31, 2049, 151936])
@pytest.mark.parametrize("top_k", [0, 50])
@pytest.mark.parametrize("masked", [False, True])
def test_infinite_temperature_draws_evenly_among_the_kept_words(vocab, top_k, masked):
    """Every weight is 1 then, and the sums are counts, exact in fp32: the token is the kept word of rank floor(u * n), but
    for the rounding of u * n itself (half a unit in the last place, below 0.01 of a word at these sizes)."""
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(vocab + top_k)
    logits = torch.randn(40, vocab, generator=g) * 3.0
    if masked:
        logits[:, 1::3] = float("-inf")
    u = torch.rand(40, generator=g)
    got = sampling.sample(logits.cuda(), float("inf"), top_k, u=u.cuda()).cpu()
    for b in range(40):
        row = logits[b]
        kept = (row > float("-inf")).nonzero().flatten()
        if 0 < top_k < vocab:
            kept = kept[row[kept] >= row.topk(top_k).values[-1]]
        rank = (kept == int(got[b])).nonzero()
        assert rank.numel() == 1, f"row {b}: token {int(got[b])} is not among the kept words"
        want = float(u[b].double()) * len(kept)
        assert int(rank) - 0.01 <= want <= int(rank) + 1.01
    ref = sampling.sample_reference(logits, float("inf"), top_k, u)
    assert int((ref != got).sum()) <= 1


@pytest.mark.parametrize("vocab,batch", [(256, 20000), (5000, 1000), (151936, 30)])
def test_a_word_without_weight_is_never_drawn(vocab, batch):
    """Half of the words are masked, and the uniform numbers lie on the first boundaries of the row's own prefix sums and a few units
    in the last place beside them, where the order of the additions decides on which side a target falls: a masked word must
    not get it."""
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(batch, vocab, generator=g)
    logits[torch.rand(batch, vocab, generator=g) < 0.5] = float("-inf")
    w = torch.where(logits > float("-inf"), torch.exp((logits - logits.amax(dim=-1, keepdim=True)) / 0.9), torch.zeros(()))
    cdf = w.double().cumsum(dim=-1)
    cdf /= cdf[:, -1:].clone()
    dev = logits.cuda()
    for trial in range(3):
        u = cdf.gather(1, torch.randint(1, 64, (batch, 1), generator=g))[:, 0].float()
        for ulps in range(-12, 13):
            got = sampling.sample(dev, 0.9, 0, u=(u * (1.0 + ulps * 2.0 ** -24)).cuda()).cpu()
            bad = (logits.gather(1, got[:, None])[:, 0] == float("-inf")).nonzero().flatten().tolist()
            assert not bad, f"trial {trial}: {len(bad)} rows drew masked words: row {bad[0]}, word {int(got[bad[0]])}"


@pytest.mark.parametrize("vocab", [31, 2049, 151936])
@pytest.mark.parametrize("top_k", [0, 50])
def test_numbers_that_are_no_draw_give_the_argmax(vocab, top_k):
    """A uniform number outside [0, 1) and a row with an infinite logit or a NaN have no draw: the arg-max of the numbers."""
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(6, vocab, generator=g)
    u = torch.tensor([-0.25, 1.0, 1.5, float("nan"), 0.5, 0.5])
    want = logits.argmax(dim=-1)
    logits[4, [7, 20]] = float("inf")
    want[4] = 7
    logits[5, int(want[5]) - 1] = float("nan")
    out = torch.full((6,), -1, dtype=torch.int64, device="cuda")
    assert sampling.sample(logits.cuda(), 0.9, top_k, u=u.cuda(), out=out).tolist() == want.tolist()


@pytest.mark.parametrize("batch,vocab,top_k", [(1, 151936, 50), (5, 151936, 200), (16, 50001, 20), (36, 151936, 50), (37, 151936, 50), (37, 151936, 0),
                                               (64, 151936, 0), (64, 1001, 0), (149, 50001, 0), (149, 50001, 7), (2, 1030, 1029)])
@pytest.mark.parametrize("temperature", [0.5, 1e-3, 1e30])
def test_draws_over_every_number_of_blocks_a_row(batch, vocab, top_k, temperature):
    """Rows whose largest words, masked words and ties lie in different blocks of a cluster: the chosen word is kept and its interval of the exact
    distribution holds u."""
    from qwen3mk import sampling

    g = torch.Generator().manual_seed(batch + vocab + top_k)
    logits = torch.randn(batch, vocab, generator=g) * 4.0
    logits[:, : vocab // 3] = float("-inf")              # whole blocks without a weight
    logits[::2, vocab // 2] = logits[::2, -1]            # equal words far apart
    u = torch.rand(batch, generator=g)
    u[0] = 0.0
    got = sampling.sample(logits.cuda(), temperature, top_k, u=u.cuda()).cpu()
    rows = logits.double()
    keep = rows > float("-inf")
    if 0 < top_k < vocab:
        keep &= rows >= rows.topk(top_k, dim=-1).values[:, -1:]
    w = torch.where(keep, torch.exp((rows - rows.max(dim=-1, keepdim=True).values) / temperature), torch.zeros_like(rows))
    cdf = (w / w.sum(dim=-1, keepdim=True)).cumsum(dim=-1)
    for b in range(batch):
        j = int(got[b])
        assert bool(keep[b, j]) and float(w[b, j]) > 0.0, (b, j)
        lo = float(cdf[b, j - 1]) if j else 0.0
        assert lo - CDF_TOL <= float(u[b]) <= float(cdf[b, j]) + CDF_TOL, (b, j, float(u[b]), lo, float(cdf[b, j]))


@pytest.mark.parametrize("batch,top_k", [(15, 120), (36, 120), (36, 121), (37, 228), (64, 228), (64, 229), (65, 228), (65, 229), (37, 0), (64, 0), (65, 0)])
@pytest.mark.parametrize("vocab", [151936, 151933])
def test_rows_that_are_read_twice(batch, top_k, vocab):
    """Clusters of two and four blocks whose threads re-read the row, on both sides of the rules (blocks an SM: 64 rows; a lane a group: twelve times the
    10 or 19 groups of a run), the largest words of some rows side by side in one warp's run or at the very end.  fp64 rule, as above."""
    from qwen3mk import sampling

    g = torch.Generator(device="cuda").manual_seed(batch + top_k)
    logits = torch.randn(batch, vocab, generator=g, device="cuda") * 3.0
    logits[1, 5000:5000 + 4 * max(top_k, 30):4] += 30.0       # every lane of a warp has candidates
    logits[2, -top_k - 5:] += 30.0
    logits[3, 7000] = float("nan")
    u = torch.rand(batch, generator=g, device="cuda")
    got = sampling.sample(logits, 0.9, top_k, u=u).tolist()
    assert got == sampling.sample(logits, 0.9, top_k, u=u).tolist()
    logits[3] = torch.where(logits[3].isnan(), float("-inf"), logits[3])
    assert got[3] == int(logits[3].argmax())                    # (a row with a NaN is not drawn from)
    keep = logits.double() > float("-inf")
    if top_k:
        keep &= logits >= logits.topk(top_k, dim=-1).values[:, -1:]
    w = torch.where(keep, torch.exp((logits.double() - logits.double().max(dim=-1, keepdim=True).values) / 0.9), 0.0)
    cdf = (w / w.sum(dim=-1, keepdim=True)).cumsum(dim=-1).cpu()
    for b in range(batch):
        j = got[b]
        lo = float(cdf[b, j - 1]) if j else 0.0
        assert bool(keep[b, j]) and (b == 3 or lo - CDF_TOL <= float(u[b]) <= float(cdf[b, j]) + CDF_TOL), (b, j)


def block_ends(vocab, blocks):
    """Where the kernel's blocks end that share a row: 32 warps a block, a run of whole groups of 128 words a warp."""
    run = (-(-vocab // (blocks * 32)) + 127) // 128 * 128
    return [min(vocab, (r + 1) * 32 * run) for r in range(blocks)]


def beside(u, ulps=range(-8, 9)):
    """Uniform numbers a few units in the last place around u, all in [0, 1)."""
    return [(u.double() * (1.0 + n * 2.0 ** -24)).float().clamp(0.0, 1.0 - 2.0 ** -24) for n in ulps]


@pytest.mark.parametrize("batch,blocks", [(4, 16), (14, 8), (36, 4), (64, 2)])
@pytest.mark.parametrize("top_k", [2, 20, 50, 200])
@pytest.mark.parametrize("part", [10, 4])
def test_a_word_that_is_not_kept_is_never_drawn(batch, blocks, top_k, part):
    """The k largest words lie in the first tenth or quarter of the row, so most of its blocks keep none, and the uniform numbers lie on the
    ends of the blocks' shares of the distribution, a few units in the last place beside them, and at both ends of [0, 1)."""
    from qwen3mk import sampling

    vocab = 151936
    g = torch.Generator(device="cuda").manual_seed(1000 * batch + 10 * top_k + part)
    logits = torch.randn((batch, vocab), generator=g, device="cuda") * 3.0
    logits[:, vocab // part:] -= 30.0
    rows = logits.double()
    keep = rows >= rows.topk(top_k, dim=-1).values[:, -1:]
    assert not bool(keep[:, vocab // part:].any())
    w = torch.where(keep, torch.exp((rows - rows.amax(dim=-1, keepdim=True)) / 0.8), torch.zeros_like(rows))
    cdf = w.cumsum(dim=-1)
    ends = (cdf / cdf[:, -1:])[:, [e - 1 for e in block_ends(vocab, blocks)]]
    zero = torch.zeros(batch, device="cuda")
    for u in [zero] + [v for r in range(blocks) for v in beside(ends[:, r])]:
        got = sampling.sample(logits, 0.8, top_k, u=u)
        bad = (~keep.gather(1, got[:, None])[:, 0]).nonzero().flatten().tolist()
        assert not bad, f"{len(bad)} rows drew words that are not kept: row {bad[0]}, word {int(got[bad[0]])}, u = 1 - {(1 - float(u[bad[0]])) * 2 ** 24} / 2^24"


@pytest.mark.parametrize("batch,blocks", [(4, 16), (14, 8), (36, 4), (64, 2), (149, 1)])
def test_a_word_whose_weight_underflows_is_never_drawn(batch, blocks):
    """Whole vocabulary, u = 0, low temperature: the first block's largest word weighs about the smallest number there is beside the row's maximum,
    the thousands of words before it weigh nothing each, although their sum under the block's own maximum does weigh something."""
    from qwen3mk import sampling

    vocab, temperature = 151936, 0.01
    end = block_ends(vocab, blocks)[0]
    gap = torch.linspace(0.95, 1.03, batch)
    logits = torch.full((batch, vocab), -5.0)
    logits[:, : end // 2] = -gap[:, None] - 0.1                 # exp(-105) and less: below half of the smallest denormal, exp(-103.28)
    logits[torch.arange(batch), torch.randint(end // 2, end, (batch,), generator=torch.Generator().manual_seed(batch))] = -gap
    logits[:, -1] = 0.0
    got = sampling.sample(logits.cuda(), temperature, 0, u=torch.zeros(batch, device="cuda")).cpu()
    # (0.25: rounding of (logit - maximum) / temperature, and of the exponential's argument)
    nats = -logits.gather(1, got[:, None])[:, 0] / temperature
    assert float(nats.max()) <= 103.28 + 0.25, nats.tolist()


@pytest.mark.parametrize("batch,blocks", [(4, 16), (14, 8), (36, 4), (64, 2), (149, 1)])
@pytest.mark.parametrize("top_k", [20, 50, 200])
def test_the_same_numbers_draw_the_same_words(batch, blocks, top_k):
    """The uniform numbers lie on boundaries between kept words and a few units in the last place beside them, where the order of the additions
    decides: every run draws the same."""
    from qwen3mk import sampling

    vocab = 151936
    g = torch.Generator(device="cuda").manual_seed(batch + top_k)
    logits = torch.randn((batch, vocab), generator=g, device="cuda") * 3.0
    rows = logits.double()
    keep = rows >= rows.topk(top_k, dim=-1).values[:, -1:]
    w = torch.where(keep, torch.exp((rows - rows.amax(dim=-1, keepdim=True)) / 0.8), torch.zeros_like(rows))
    cdf = w.cumsum(dim=-1)
    cdf /= cdf[:, -1:].clone()
    kept = [torch.nonzero(keep[b]).flatten() for b in range(batch)]
    for trial in range(8):
        edge = torch.stack([cdf[b, kept[b][(7 * trial + b) % (len(kept[b]) - 1)]] for b in range(batch)])
        for u in beside(edge, range(-4, 5)):
            want = sampling.sample(logits, 0.8, top_k, u=u)
            again = torch.stack([sampling.sample(logits, 0.8, top_k, u=u) for _ in range(6)])
            assert bool((again == want).all()), f"trial {trial}: rows {(again != want).any(0).nonzero().flatten().tolist()}"
