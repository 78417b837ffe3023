"""Search paths of the sampler kernels at the sizes where they can go wrong: the CPU oracle, fed the kernel's own fp32
probabilities and RNG states, must land on the same bits (threshold, totals, weights, id)."""
import numpy as np
import pytest
import torch

from helpers import make_logits
from oracle import c_oracle as co

pytestmark = pytest.mark.gpu

FIELDS_U = ("left", "seqk", "sgtk", "rounds", "idxt", "early_exit")
FIELDS_F = ("threshold", "comp", "sgtp", "sum_p", "randp", "sum_o", "rand2", "pmin", "pmax")


def check_against_oracle(abi, lg, seed, temp, k, p, mode=0, pen=None, rows=4, decay=0.95):
    B, V = lg.shape
    st = abi.setup_rand(seed, B)
    st_cpu = st.cpu().numpy().copy()
    pen_dev = pen.clone().cuda() if pen is not None else None
    abi.set_path(mode)
    try:
        out, probs, tr = abi.sample(lg.cuda(), st, temp, k, p, penalties=pen_dev, presence=0.1, repetition=0.1, decay=decay, debug=True)
    finally:
        abi.set_path(0)
    knd, scale, kk, pp = co.normalise(V, B, 1, temp, k, p, with_penalties=pen is not None)
    for b in (range(B) if rows >= B else sorted({0, B - 1, B // 2, B // 3})[:rows]):
        pen_cpu = pen[b].numpy().copy() if pen is not None else None
        tok, o, _ = co.sample_row(lg[b].numpy(), st_cpu[64 * b:64 * b + 64], knd, scale, kk, pp, penalties=pen_cpu, presence=0.1,
                                  repetition=0.1, decay=decay, probs_in=probs[b].cpu().numpy())
        g = tr[b]
        assert tok == int(out[b]) == g.token, b
        for f in FIELDS_U:
            assert getattr(o, f) == getattr(g, f), (b, f, getattr(o, f), getattr(g, f))
        for f in FIELDS_F:
            x, y = np.float32(getattr(o, f)), np.float32(getattr(g, f))
            assert x.view(np.uint32) == y.view(np.uint32), (b, f, x, y)
        if pen is not None:
            assert np.array_equal(pen_cpu, pen_dev[b].cpu().numpy(), equal_nan=True)
            assert np.array_equal(np.signbit(pen_cpu[pen_cpu == 0]), np.signbit(pen_dev[b].cpu().numpy()[pen_cpu == 0]))
    assert abi.device_status() == 0
    return tr


@pytest.mark.parametrize("mode", [0, 2, 3, 4])        # the planner's choice, streaming, on-chip, one CTA per row
@pytest.mark.parametrize("kind,B,V,temp", [("normal3", 3, 4, 1.0), ("peaked", 130, 4096, 1.0), ("uniform", 4, 4100, 0.7),
                                           ("coarse", 300, 8188, 1.0), ("special", 5, 50304, 1.3), ("equal", 4, 8192, 1.0),
                                           ("normal3", 2, 65536, 0.02)])
def test_rows_of_which_nothing_is_cut_off(abi, mode, kind, B, V, temp):
    """No top_k and top_p = 1: the recount runs on probabilities that are never stored (and, at temperature 0.02, on
    numerators too small for the short division)."""
    tr = check_against_oracle(abi, make_logits(kind, B, V, 11, torch), 5, temp, -1, 1.0, mode)
    assert all(t.rounds == 0 for t in tr)
    if mode in (0, 4):
        pen = torch.rand(B, V, generator=torch.Generator().manual_seed(1)) * 0.5
        check_against_oracle(abi, make_logits(kind, B, V, 12, torch), 6, temp, -1, 1.0, mode, pen=pen)


@pytest.mark.parametrize("mode", [2, 3, 4, 5, 6])    # streaming, on-chip, one CTA per row; exact search only in the last two
@pytest.mark.parametrize("kind,V,k,p", [("normal3", 4, -1, 0.5), ("uniform", 28, 5, 0.9), ("coarse", 64, -1, 0.6), ("equal", 508, 40, 0.3),
                                        ("uniform", 512, -1, 0.95), ("coarse", 512, 100, 1.0), ("uniform", 516, 200, 0.99),
                                        ("peaked", 50304, 1, 1.0), ("normal3", 100256, 50, 1e-7), ("coarse", 32768, 250, 0.9)])
def test_integer_search_by_rank(abi, mode, kind, V, k, p):
    """Candidate lists shorter than the sample, around the longest length, made of few distinct values, all equal, cut by the
    count alone, and a top_p inside the margin of the empty set."""
    for seed in (1, 2):
        check_against_oracle(abi, make_logits(kind, 6, V, seed, torch), seed, 0.9, k, p, mode)


@pytest.mark.parametrize("mode,rep,longest", [(2, False, 512), (3, True, 512), (4, True, 512), (4, False, 1024)])
def test_longest_list_of_the_integer_search(abi, mode, rep, longest):
    """Rows whose list is the whole row, of just under, exactly and just over the longest length: settled on integer masses
    up to it, by the exact search beyond.  (One CTA per row without penalties holds twice the length.)"""
    for V in (longest - 4, longest, longest + 4):
        pen = torch.rand(6, V, generator=torch.Generator().manual_seed(4)) * 0.5 if rep else None
        tr = check_against_oracle(abi, make_logits("uniform", 6, V, 71, torch), 3, 0.9, -1, 0.95, mode, pen=pen, rows=6)
        for t in tr:
            assert t.ncand == V and t.path == 0
            outcome, rounds = (t.t_ns[0] >> 16) & 0xf, t.t_ns[0] & 0xffff
            assert (outcome, rounds > 0) == ((1, False) if V <= longest else (0, True)), (V, outcome, rounds)
            if mode == 4:
                assert (t.t_ns[0] >> 20) & 1 == (1 if V <= longest else 0)


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 5, 6])  # the planner's choice, whole row only, streaming, on-chip; exact search only
@pytest.mark.parametrize("kind,B,V,temp,k,p", [("normal3", 2, 16384, 1.0, -1, 0.9), ("normal3", 3, 16388, 1.0, -1, 0.99),
                                               ("peaked", 130, 50304, 1.0, -1, 0.95), ("uniform", 2, 131072, 1.0, -1, 0.5),
                                               ("uniform", 4, 20484, 0.7, -1, 0.999999), ("normal3", 3, 65536, 0.8, 1000, 0.95),
                                               ("coarse", 3, 50304, 0.9, 3000, 0.99), ("coarse", 2, 32768, 1.0, -1, 0.6),
                                               ("special", 3, 50304, 1.3, 700, 0.9), ("normal3", 2, 65536, 0.02, 300, 0.9999),
                                               ("uniform4", 2, 8192, 1.0, 8191, 1.0), ("normal3", 2, 16384, 1.0, -1, 1e-46),
                                               ("equal", 2, 32768, 1.0, 500, 0.9)])
def test_wide_kept_sets(abi, mode, kind, B, V, temp, k, p):
    """Cutoffs far down the row: lists collected again under a bound read off the histogram, long lists, and whole rows, all
    searched by evaluating points of the kernel's own choice; ties, counts met exactly, zero probabilities, and a top_p
    that is zero in fp32."""
    check_against_oracle(abi, make_logits(kind, B, V, 21, torch), 9, temp, k, p, mode)
    if B <= 4 and mode != 1:
        pen = torch.rand(B, V, generator=torch.Generator().manual_seed(2)) * 0.5
        check_against_oracle(abi, make_logits(kind, B, V, 22, torch), 10, temp, k, p, mode, pen=pen)


@pytest.mark.parametrize("mode", [0, 2, 3, 4])
@pytest.mark.parametrize("B,V,density,decay", [(3, 50304, 0.004, 0.95), (130, 4100, 0.0, 0.5), (4, 300000, 0.001, -0.5),
                                               (150, 32768, 0.02, 0.95), (2, 16384, 0.1, float("inf")), (5, 65536, 1.0, 0.95)])
def test_zero_penalties_are_neither_copied_nor_rewritten(abi, mode, B, V, density, decay):
    """Groups whose penalties are all +0 are left alone; -0 becomes +0, a zero times an infinite decay NaN, and the sampled id
    gets its presence penalty wherever it lies."""
    g = torch.Generator().manual_seed(3)
    pen = torch.rand(B, V, generator=g) * (torch.rand(B, V, generator=g) < density)
    pen[:, 5::97] *= -0.0
    pen[0] = 0.0
    tr = check_against_oracle(abi, make_logits("peaked", B, V, 31, torch), 7, 0.8, 50, 0.9, mode, pen=pen, decay=decay)
    assert all(0 <= t.token < V for t in tr)


@pytest.mark.parametrize("mode", [0, 2, 3, 4, 6])     # the planner's choice, streaming, on-chip, one CTA per row, exact search only
@pytest.mark.parametrize("V,low,near,top", [(6144, 6024, 100, 20), (8192, 7282, 900, 10), (12000, 11800, 180, 20), (30000, 29300, 690, 10)])
def test_elements_above_the_bound_whose_quotients_tie_with_it(abi, mode, V, low, near, top):
    """Rows of a few large logits, some that lie one to three floats above the rest, and the rest: the bound of the candidate
    list falls on the rest, more than top_k elements lie above it, and after the division by the denominator many of those tie
    with it, so that the cutoff is the bound's own probability."""
    B, k = 48, 50
    rng = np.random.default_rng(V + near)
    lg = np.empty((B, V), np.float32)
    for b in range(B):
        x = np.float32(rng.uniform(-1.0, 1.0))
        rest = np.full(V, x, np.float32)
        up = x
        for _ in range(1 + b % 3):
            up = np.nextafter(up, np.float32(4))
            rest[low:low + near][rng.random(near) < (1.0 if up == np.nextafter(x, np.float32(4)) else 0.5)] = up
        rest[low + near:] = np.float32(x + rng.uniform(0.5, 1.0))
        lg[b] = rng.permutation(rest)
    check_against_oracle(abi, torch.from_numpy(lg), 3, 1.0, k, 1.0, mode, rows=B)


@pytest.mark.parametrize("kind,B,V,p,mode", [("head", 32, 1048576, 0.95, 0), ("head", 64, 151936, 0.9, 0), ("head", 64, 151936, 0.95, 0),
                                             ("head", 128, 50304, 0.95, 0), ("head", 4, 131072, 0.95, 0), ("head", 16, 32000, 0.95, 0),
                                             ("normal3", 4, 151936, 0.9, 2), ("normal3", 4, 50304, 0.95, 2)])
def test_lowered_bound_gives_a_list_that_settles_the_row(abi, kind, B, V, p, mode):
    """Rows whose first list is too thin: a wide head (1 % of the ids raised by 8, nothing else within ten octaves of them)
    and normal rows.  The list collected again must hold enough and fit, so that no row is searched whole."""
    if kind == "head":
        g = torch.Generator(device="cuda").manual_seed(4)
        lg = torch.randn(B, V, generator=g, device="cuda")
        ids = torch.stack([torch.randperm(V, generator=g, device="cuda")[:V // 100] for _ in range(B)])
        lg = lg.scatter_add_(1, ids, torch.full(ids.shape, 8.0, device="cuda")).cpu()
    else:
        lg = make_logits(kind, B, V, 41, torch)
    tr = check_against_oracle(abi, lg, 11, 1.0, -1, p, mode, rows=3)
    assert [t.path for t in tr] == [0] * B


@pytest.mark.parametrize("mode", [0, 2, 6])           # the planner's choice, streaming, exact search only
@pytest.mark.parametrize("kind,V,p", [("uniform", 4096, 0.5), ("uniform", 4100, 0.5), ("coarse", 4096, 0.6), ("coarse", 4100, 0.6),
                                      ("normal3", 20480, 0.9), ("normal3", 32000, 0.9), ("normal3", 50304, 0.9)])
def test_list_lengths_around_the_line_between_the_two_searches(abi, mode, kind, V, p):
    """Lists of 513 to about 7000 entries, on both sides of the 4096 up to which the reference's own pivots are evaluated."""
    tr = check_against_oracle(abi, make_logits(kind, 12, V, 51, torch), 13, 1.0, -1, p, mode, rows=12)
    assert any(t.path == 0 and t.ncand > 512 for t in tr)
