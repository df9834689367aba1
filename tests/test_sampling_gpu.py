"""The sampling kernel: greedy with ties, log-probabilities, the seeded draw against the
plain restatement, empirical frequencies against the exact warped distribution
(cases of the reference's tests/cuda/test_sampling.cu:84-161)."""

import numpy as np
import pytest
import torch

import plain_llama as P
from redline_b200.ops import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(logits, temperature, top_k, top_p, seeds, positions, two_stage=None):
    """two_stage None: both ways must agree (greedy rows take the two-stage arg max when scratch is given)."""
    if two_stage is None:
        a = run(logits, temperature, top_k, top_p, seeds, positions, two_stage=False)
        b = run(logits, temperature, top_k, top_p, seeds, positions, two_stage=True)
        assert np.array_equal(a[0], b[0]) and np.abs(a[1] - b[1]).max() < 1e-4
        return b
    R = logits.shape[0]
    f = lambda v, dt: torch.tensor(np.broadcast_to(np.asarray(v), (R,)).copy(), dtype=dt, device=DEV)  # noqa: E731
    seeds = np.broadcast_to(np.asarray(seeds, dtype=np.uint64), (R,))
    lo = torch.tensor((seeds & 0xFFFFFFFF).astype(np.int64), device=DEV).to(torch.int32)
    hi = torch.tensor((seeds >> 32).astype(np.int64), device=DEV).to(torch.int32)
    tok = torch.empty(R, dtype=torch.int32, device=DEV)
    lp = torch.empty(R, dtype=torch.float32, device=DEV)
    scratch = torch.full((R * kernels.SAMPLE_CHUNKS * 4,), float("nan"), device=DEV) if two_stage else None
    kernels.sample(logits, R, f(temperature, torch.float32), f(top_k, torch.int32), f(top_p, torch.float32),
                   lo, hi, f(positions, torch.int32), tok, lp, scratch=scratch)
    return tok.cpu().numpy(), lp.cpu().numpy()


def test_greedy_ties_and_logprobs():
    V = 1000
    l = torch.randn(12, V, device=DEV)
    l[3, 17] = l[3, 900] = l[3].max() + 1.0          # a tie: the smaller index wins
    l[5, 0] = 50.0
    tok, lp = run(l, 0.0, 0, 1.0, 0, 0)
    ref = l.double().cpu()
    assert tok.tolist() == [int(ref[i].argmax()) if i != 3 else 17 for i in range(12)]
    want = torch.log_softmax(ref, -1)[torch.arange(12), torch.tensor(tok.astype(np.int64))]
    assert np.abs(lp - want.numpy()).max() < 1e-4
    # 16 rows and more: the first stage cuts a row into fewer, longer pieces (and marks the unused slots
    # empty); a vocabulary that is no multiple of anything, a tie across two pieces, a maximum in the last one
    for V, R in [(128256, 16), (331, 20), (50001, 33)]:
        l = torch.randn(R, V, device=DEV)
        l[1, 5] = l[1, V - 2] = l[1].max() + 2.0
        l[2, V - 1] = 40.0
        tok, lp = run(l, 0.0, 0, 1.0, 0, 0)
        ref = l.double().cpu()
        assert tok.tolist() == [int(ref[i].argmax()) if i != 1 else 5 for i in range(R)]
        want = torch.log_softmax(ref, -1)[torch.arange(R), torch.tensor(tok.astype(np.int64))]
        assert np.abs(lp - want.numpy()).max() < 1e-4


@pytest.mark.parametrize("T,k,p", [(1.0, 0, 1.0), (0.7, 5, 1.0), (1.3, 0, 0.8), (0.9, 20, 0.6)])
def test_seeded_draw_equals_the_plain_restatement(T, k, p):
    V = 331
    l = (torch.randn(40, V) * 2).float()
    pos = np.arange(40) + 3
    tok, _ = run(l.to(DEV), T, k, p, 1234567890123, pos)
    for r in range(40):
        assert tok[r] == P.gumbel_draw(l[r].numpy(), T, k, p, 1234567890123, int(pos[r])), r
    tok2, _ = run(l.to(DEV), T, k, p, 1234567890123, pos)
    assert np.array_equal(tok, tok2)
    # a row's draw depends on (seed, position), not on where the row sits in the batch
    perm = np.random.RandomState(0).permutation(40)
    tok3, _ = run(l[perm].to(DEV), T, k, p, 1234567890123, pos[perm])
    assert np.array_equal(tok3, tok[perm])


@pytest.mark.parametrize("T,k,p", [(1.0, 0, 1.0), (0.7, 4, 1.0), (1.5, 0, 0.7), (0.8, 6, 0.9)])
def test_frequencies_follow_the_warped_distribution(T, k, p):
    V, R = 16, 6000
    row = np.array([2.0, 1.5, 1.5, 1.0, 0.7, 0.3, 0.0, -0.2, -0.5, -1.0, -1.0, -2.0, -3.0, -3.5, -5.0, -8.0],
                   dtype=np.float32)
    l = torch.tensor(np.tile(row, (R, 1)), device=DEV)
    tok, _ = run(l, T, k, p, 99, np.arange(R))
    want = P.warped_distribution(row, T, k, p)
    freq = np.bincount(tok, minlength=V) / R
    assert np.all(freq[want == 0] == 0), "a token outside the kept set was drawn"
    assert np.abs(freq - want).max() < 0.025


def test_large_vocabulary_top_k_membership():
    V = 128256
    l = torch.randn(4, V, device=DEV)
    tok, lp = run(l, 1.0, 50, 1.0, [1, 2, 3, 4], [10, 10, 10, 10])
    top = torch.topk(l, 50, dim=-1).indices.cpu().numpy()
    assert all(tok[r] in top[r] for r in range(4)) and np.all(np.isfinite(lp))
    tok_g, lp_g = run(l, 0.0, 0, 1.0, 0, 0)
    assert tok_g.tolist() == l.argmax(-1).tolist()
    want = torch.log_softmax(l.double(), -1).max(-1).values.cpu().numpy()
    assert np.abs(lp_g - want).max() < 1e-4
    # greedy and sampled rows in one launch
    temp = np.array([0.0, 1.0, 0.0, 0.7], dtype=np.float32)
    tok_m, _ = run(l, temp, 50, 1.0, [1, 2, 3, 4], [10, 10, 10, 10])
    assert tok_m[0] == tok_g[0] and tok_m[2] == tok_g[2] and tok_m[1] in top[1] and tok_m[3] in top[3]


@pytest.mark.parametrize("V,ld", [(8192, 8192), (8203, 8203), (8203, 8208), (20001, 20004)])
@pytest.mark.parametrize("T,k,p", [(1.0, 7, 1.0), (0.7, 0, 0.05), (1.3, 50, 0.6), (0.9, 1, 1.0), (2.0, 8191, 1e-6)])
def test_draw_over_a_cluster_equals_the_plain_restatement(V, ld, T, k, p):
    """Rows cut over a cluster of CTAs (large vocabularies): the last CTA's share is short or ragged, rows start off
    16-byte boundaries, logits tie at the thresholds and across shares, others are -inf, one row is greedy."""
    rng = np.random.RandomState(V + k)
    l = (rng.randn(5, V) * 3).astype(np.float32)
    l[1] = np.round(l[1])                                  # many ties at every threshold
    l[2, rng.rand(V) < 0.9] = -np.inf
    l[3, V - 1] = l[3, 0] = l[3].max() + 1.0               # the maximum twice, in the first and the last share
    buf = torch.full((5, ld), float("nan"), device=DEV)
    buf[:, :V] = torch.from_numpy(l).to(DEV)
    temp = np.array([T, T, T, T, 0.0], dtype=np.float32)
    tok, lp = run(buf[:, :V], temp, k, p, 1234567890123, np.arange(5) + 3)
    for r in range(4):
        assert tok[r] == P.gumbel_draw(l[r], T, k, p, 1234567890123, r + 3), r
    assert tok[4] == int(l[4].argmax())
    want = torch.log_softmax(torch.from_numpy(l).double(), -1)[torch.arange(5), torch.from_numpy(tok.astype(np.int64))]
    assert np.abs(lp - want.numpy()).max() < 1e-4


@pytest.mark.parametrize("V", [8192, 20001, 128256])
def test_the_kernels_draw_the_same(V):
    """What the caller says about the rows decides which kernel runs, at row counts on both sides of the lines; the draws
    are the same, also where what it says is wrong."""
    R = 70
    l = torch.randn(R, V, device=DEV) * 3
    i32 = lambda v: torch.full((R,), v, dtype=torch.int32, device=DEV)      # noqa: E731
    temp = torch.full((R,), 0.8, device=DEV)
    temp[::3] = 0.0
    seed, pos = torch.arange(R, dtype=torch.int32, device=DEV), i32(9)
    scratch = torch.empty(R * kernels.SAMPLE_CHUNKS * 4, device=DEV)
    assert not kernels.sample_clusters(1, V, kernels.DRAWS_NONE) and kernels.sample_clusters(70, V, kernels.DRAWS_FILTERED)
    assert kernels.sample_clusters(70, V, kernels.DRAWS_PLAIN) == (V == 128256)
    assert not kernels.sample_clusters(1, 8191, kernels.DRAWS_FILTERED)
    for k, p in ((0, 1.0), (40, 0.9)):
        got = []
        for draws in (kernels.DRAWS_NONE, kernels.DRAWS_PLAIN, kernels.DRAWS_FILTERED):
            tok, lp = i32(-1), torch.empty(R, device=DEV)
            kernels.sample(l, R, temp, i32(k), torch.full((R,), p, device=DEV), seed, i32(0), pos, tok, lp, scratch=scratch,
                           draws=draws)
            got.append((tok, lp))
        assert all(torch.equal(t, got[0][0]) and (x - got[0][1]).abs().max() < 1e-4 for t, x in got)
        assert torch.equal(got[0][0][::3], l.argmax(-1).int()[::3])


@pytest.mark.parametrize("T,k,p", [(1.0, 0, 0.95), (1.4, 200, 0.9), (3.0, 40000, 0.8)])
def test_draw_at_a_served_vocabulary(T, k, p):
    """128,256 logits, 64 KB of a row to a CTA (more than a kernel has without asking): tokens drawn from flat and from
    peaked rows, which are not the arg max."""
    V = 128256
    rng = np.random.RandomState(int(10 * T))
    l = (rng.randn(4, V) * np.array([[0.1], [1.0], [2.5], [1.0]])).astype(np.float32)
    l[3] = np.round(4 * l[3]) / 4                          # ties at every threshold
    tok, lp = run(torch.from_numpy(l).to(DEV), T, k, p, 987654321, np.arange(4) + 11)
    want = [P.gumbel_draw(l[r], T, k, p, 987654321, r + 11) for r in range(4)]
    assert tok.tolist() == want and sum(int(l[r].argmax()) != want[r] for r in range(4)) >= 3
    full = torch.log_softmax(torch.from_numpy(l).double(), -1)[torch.arange(4), torch.tensor(want)]
    assert np.abs(lp - full.numpy()).max() < 1e-4


@pytest.mark.parametrize("two_stage", [False, True])
@pytest.mark.parametrize("V", [1, 331, 8191, 8192, 20001, 128256])
def test_rows_without_a_best_logit(V, two_stage):
    """Rows of NaN and of -inf only, greedy and sampled (in one block and over a cluster): token 0 and a NaN
    log-probability; the rows beside them are drawn as ever."""
    l = torch.randn(6, V, device=DEV)
    l[0], l[1], l[3], l[4] = float("nan"), -float("inf"), float("nan"), -float("inf")
    temp = np.array([0.0, 0.0, 0.0, 0.8, 0.8, 0.8], dtype=np.float32)
    tok, lp = run(l, temp, 5 if V > 5 else 0, 0.9, 7, np.arange(6), two_stage)
    assert tok[[0, 1, 3, 4]].tolist() == [0] * 4 and np.isnan(lp[[0, 1, 3, 4]]).all()
    assert tok[2] == int(l[2].argmax()) and np.isfinite(lp[[2, 5]]).all()
    assert tok[5] == P.gumbel_draw(l[5].cpu().numpy(), 0.8, 5 if V > 5 else 0, 0.9, 7, 5)


@pytest.mark.parametrize("V", [1, 511, 4096, 50001])
def test_gather_logprob_one_pass(V):
    """Rows shorter than a block's first loads, on its edge, and ragged; values far apart and -inf."""
    l = torch.randn(3, V, device=DEV) * 30
    if V > 1:
        l[1, ::2] = -float("inf")
    l[2] -= 1e4
    tgt = torch.tensor([0, V // 2 | 1 if V > 1 else 0, V - 1], device=DEV, dtype=torch.int32).clamp(max=V - 1)
    out = torch.empty(3, device=DEV)
    kernels.gather_logprob(l, 3, tgt, out)
    want = torch.log_softmax(l.double(), -1)[torch.arange(3), tgt.long()]
    fine = torch.isfinite(want)          # (float32 sums of values about 1e4: a unit in the last place is 1e-3)
    assert torch.equal(torch.isfinite(out), fine) and (out.double() - want)[fine].abs().max().item() < 2e-3


def test_gather_logprob():
    l = torch.randn(9, 777, device=DEV) * 3
    tgt = torch.randint(0, 777, (9,), device=DEV, dtype=torch.int32)
    out = torch.empty(9, device=DEV)
    kernels.gather_logprob(l, 9, tgt, out)
    want = torch.log_softmax(l.double(), -1)[torch.arange(9), tgt.long()]
    assert (out.double() - want).abs().max().item() < 1e-4
