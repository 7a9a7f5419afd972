"""GPU parity of the streamed window kernel (Moe for windows of <= 16 rows) at the edges of its cuts: k ranges of one stage
(256) and of an odd number of them, one block of columns' worth of experts, one and two member sets, repeated picks, windows
without an expert of this GPU, and both launch widths."""
import numpy as np
import pytest

from conftest import TOL, rel_err

pytestmark = pytest.mark.gpu


def run(pkg, cuda, bank, x, picks, rw, H, I, E, S, rows, synth, max_rows=None, **kw):
    import torch
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=max_rows or rows, **kw))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd = t(x.view(np.int16)).view(torch.bfloat16)
    for _ in range(2):                                   # the second launch runs on the first one's counters and words
        moe.run(bank, xd, t(picks), t(rw), rows)
    torch.cuda.synchronize()
    assert int(moe.status.cpu()[0]) == 0
    return moe.output[:rows].cpu().numpy()


@pytest.mark.parametrize("H,I,E,S,rows", [(256, 256, 3, 2, 1), (768, 256, 5, 3, 7), (512, 1280, 9, 4, 16), (2304, 768, 8, 5, 9),
                                          (1024, 512, 40, 32, 16), (256, 768, 1, 2, 8),
                                          (3328, 256, 3, 2, 3), (256, 3328, 3, 2, 10)])
def test_edges_vs_oracle(pkg, oracle, synth, cuda, H, I, E, S, rows):
    bank = synth.expert_bank(31 + H + I, H, I, E, svh_scale=True)
    x, (picks, rw) = synth.activations_bf16(32, rows, H), synth.route(33, rows, E, S - 1, shared_bias=rows > 1)
    got = run(pkg, cuda, synth.to_device(bank, cuda), x, picks, rw, H, I, E, S, rows, synth)
    want = oracle.combine(oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1), rw, rows, S, H)
    emax, erms = rel_err(got, want)
    assert np.isfinite(got).all() and emax < TOL and erms < TOL, (emax, erms)


@pytest.mark.parametrize("H,I,E,S,rows,kw", [(256, 512, 3, 3, 17, {}), (512, 512, 40, 9, 40, {}), (768, 512, 8, 2, 128, {}),
                                             (512, 512, 12, 4, 64, dict(expert_lo=1, expert_hi=9, shared_rows=(10, 50)))])
def test_short_chunks_vs_oracle(pkg, oracle, synth, cuda, H, I, E, S, rows, kw):
    # chunks of many rows an expert: the GEMMs in fine steps (40 experts: at the line, streamed); a repeated pick, a rank's share
    bank = synth.expert_bank(51 + H + rows, H, I, E, svh_scale=True)
    x, (picks, rw) = synth.activations_bf16(52, rows, H), synth.route(53, rows, E, S - 1)
    if S > 2:
        picks[3, 1] = picks[3, 0]                        # a repeated pick is not computed again
        rw[3, 1] = 0
    got = run(pkg, cuda, synth.to_device(bank, cuda), x, picks, rw, H, I, E, S, rows, synth, **kw)
    Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1).reshape(rows, S, H)
    lo, hi = kw.get("expert_lo", 0), kw.get("expert_hi", E)
    r0, r1 = kw.get("shared_rows", (0, rows))
    here = (picks >= lo) & (picks < hi) | (picks == E) & (np.arange(rows)[:, None] >= r0) & (np.arange(rows)[:, None] < r1)
    want = np.where(here[..., None], np.where((np.arange(S) == S - 1)[None, :, None], 1, rw[..., None]) * Y, 0).sum(1)
    emax, erms = rel_err(got, want)
    assert emax < TOL and erms < TOL, (emax, erms)


def launches(pkg, moe, *args):
    """Kernels of one call, counted as the nodes of its graph."""
    import torch
    cache, side = pkg.GraphCache(bounded=True), torch.cuda.Stream()
    torch.cuda.synchronize()
    cache.run(1, lambda: moe.run(*args), stream=side)
    side.synchronize()
    return cache.stats()["retained_nodes"]


@pytest.mark.parametrize("H,I,E,rows,kw", [(256, 512, 24, 17, {}), (512, 512, 24, 40, {}), (768, 256, 48, 101, {}), (512, 768, 48, 128, {}),
                                           (512, 512, 24, 40, dict(expert_lo=1, expert_hi=19, shared_rows=(10, 30)))])
def test_streamed_chunks_with_popular_experts(pkg, oracle, synth, cuda, H, I, E, rows, kw):
    # few rows an expert on average, so that the chunk is streamed, but three that most rows pick: whole sixteens of members, a remainder, one more
    # than a sixteen; and a repeated pick, which is not computed again
    import torch
    S = 4
    bank = synth.expert_bank(54 + H + rows, H, I, E, svh_scale=True)
    x, (_, rw) = synth.activations_bf16(52, rows, H), synth.route(53, rows, E, S - 1)
    rng = np.random.default_rng(55)
    picks = np.stack([np.append(8 + rng.permutation(E - 8)[:S - 1], E) for _ in range(rows)]).astype(np.int32)
    picks[:rows - 3, 0] = 5
    picks[:max(16, (rows - 4) // 16 * 16), 1] = 6
    picks[rows - 17:, 2] = 7
    picks[3, 1], rw[3, 1] = picks[3, 0], 0
    dbank = synth.to_device(bank, cuda)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=rows, **kw))
    assert launches(pkg, moe, dbank, t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw), rows) == 1
    got = run(pkg, cuda, dbank, x, picks, rw, H, I, E, S, rows, synth, **kw)
    Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1).reshape(rows, S, H)
    lo, hi = kw.get("expert_lo", 0), kw.get("expert_hi", E)
    r0, r1 = kw.get("shared_rows", (0, rows))
    here = (picks >= lo) & (picks < hi) | (picks == E) & (np.arange(rows)[:, None] >= r0) & (np.arange(rows)[:, None] < r1)
    want = np.where(here[..., None], np.where((np.arange(S) == S - 1)[None, :, None], 1, rw[..., None]) * Y, 0).sum(1)
    emax, erms = rel_err(got, want)
    assert emax < TOL and erms < TOL, (emax, erms)


@pytest.mark.parametrize("H,I,E,S,rows,kw", [(512, 512, 40, 3, 96, {}), (768, 256, 30, 2, 128, {}), (256, 512, 24, 4, 17, {}),
                                             (512, 512, 24, 4, 40, dict(expert_lo=1, expert_hi=19, shared_rows=(10, 30))),
                                             (256, 256, 300, 9, 18, {}), (256, 256, 300, 9, 40, {})])
def test_chunks_on_both_sides_of_the_line(pkg, oracle, synth, cuda, H, I, E, S, rows, kw):
    # few rows per expert: streamed, unless the tables of many experts take a CTA's room (the last one).  A row is held against both orders of
    # the oracle's sums: in row 88 of (768, 256, 30) they round a 16-bit product of 32..64 to neighbours, and differ by 2.03e-3 themselves.
    bank = synth.expert_bank(51 + H + rows, H, I, E, svh_scale=True)
    x, (picks, rw) = synth.activations_bf16(52, rows, H), synth.route(53, rows, E, S - 1)
    got = run(pkg, cuda, synth.to_device(bank, cuda), x, picks, rw, H, I, E, S, rows, synth, **kw)
    lo, hi = kw.get("expert_lo", 0), kw.get("expert_hi", E)
    r0, r1 = kw.get("shared_rows", (0, rows))
    here = (picks >= lo) & (picks < hi) | (picks == E) & (np.arange(rows)[:, None] >= r0) & (np.arange(rows)[:, None] < r1)
    scale, off = 0, []
    for mode in (0, 1):
        Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=mode).reshape(rows, S, H)
        want = np.where(here[..., None], np.where((np.arange(S) == S - 1)[None, :, None], 1, rw[..., None]) * Y, 0).sum(1)
        scale = max(scale, np.abs(want).max())
        off.append(np.abs(got - want).max(1))
    assert np.min(off, axis=0).max() < TOL * scale


@pytest.mark.parametrize("H,I,E,S", [(512, 512, 16, 7), (256, 256, 384, 9), (256, 256, 4, 3), (512, 256, 2, 2), (256, 512, 16, 17), (256, 256, 200, 11)])
def test_windows_of_large_handles(pkg, synth, cuda, H, I, E, S):
    # calls of up to 16 rows are one launch with the bytes of a handle for 16, also where the line for longer chunks is at 16 rows or fewer
    # (few experts for the slots, tables of many experts); a call of 17 rows in between
    import torch
    dbank = synth.to_device(synth.expert_bank(61 + H, H, I, E, svh_scale=True), cuda)
    x, (picks, rw) = synth.activations_bf16(62, 17, H), synth.route(63, 17, E, S - 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd, pd, wd = t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw)
    small, large = (pkg.Moe(pkg.make_config(H, I, E, S, max_rows=n)) for n in (16, 8192))
    for rows in (1, 2, 17, 9, 16):
        args = (dbank, xd[:rows], pd[:rows], wd[:rows], rows)
        large.run(*args)
        torch.cuda.synchronize()
        assert int(large.status.cpu()[0]) == 0
        if rows > 16:
            continue
        small.run(*args)
        torch.cuda.synchronize()
        assert torch.equal(large.output[:rows].view(torch.int32), small.output[:rows].view(torch.int32))
        pairs = [pkg._view(m.pairs_ptr.value, (rows * S, H), torch.int32) for m in (large, small)]
        assert torch.equal(*pairs)
        assert launches(pkg, large, *args) == launches(pkg, small, *args) == 1


@pytest.mark.parametrize("H,I,E,S,last", [(1536, 256, 30, 3, 120), (1024, 1024, 20, 5, 37), (1024, 2048, 12, 4, 24), (512, 512, 64, 3, 128)])
def test_line_between_the_kernels(pkg, synth, cuda, H, I, E, S, last):
    # one launch up to 4.5 + 3 * 2^20 / (H I) rows per routed expert, at most 8 (128 rows): small experts have the line later
    import torch
    dbank = synth.to_device(synth.expert_bank(64 + H, H, I, E, svh_scale=True), cuda)
    x, (picks, rw) = synth.activations_bf16(65, last + 1, H), synth.route(66, last + 1, E, S - 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd, pd, wd = t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw)
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=512))
    assert launches(pkg, moe, dbank, xd, pd, wd, last) == 1
    assert launches(pkg, moe, dbank, xd, pd, wd, last + 1) > 1


# members of the experts: one, and around the MMAs' and slabs' sizes of the GEMMs, of which 32, 64 and more rows have different numbers of
# partial sums on the way at once; the shared expert has all 128 rows
FINE_COUNTS = (1, 31, 32, 33, 64, 65, 96, 97, 93)


@pytest.mark.parametrize("H,I", [(256, 256), (512, 768), (768, 512), (1024, 2304), (2048, 512), (2304, 256), (3072, 256), (4096, 256), (256, 4096)])
def test_chunks_are_as_exact_as_windows(pkg, oracle, synth, cuda, H, I):
    # beyond the line a chunk of up to 128 rows goes to the GEMMs, whose sums are then chains of at most 512 k like the streamed kernel's: as near
    # to sums in 64 bits (oracle mode 1) as the same rows in windows of 16.  What separates either from those are bf16 roundings that fall the
    # other way, some hundred of a run, so the two distances agree to a tenth or so; one chain over K = 2048 is 2 to 4 times as far.
    import torch
    rows, S, E = 128, 5, len(FINE_COUNTS)
    bank = synth.expert_bank(81 + H + I, H, I, E, svh_scale=True)
    dbank = synth.to_device(bank, cuda)
    order = np.repeat(np.arange(E, dtype=np.int32), FINE_COUNTS)         # (no expert twice in a row: none has more than 128 members)
    picks = np.concatenate([order.reshape(S - 1, rows).T, np.full((rows, 1), E, np.int32)], 1).astype(np.int32)
    x, rw = synth.activations_bf16(82, rows, H), np.full((rows, S), 0.25, np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd, pd, wd = t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw)
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=rows))
    Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1).reshape(rows, S, H)

    def run(lo, n):
        moe.run(dbank, xd[lo:], pd[lo:], wd[lo:], n)
        torch.cuda.synchronize()
        assert int(moe.status.cpu()[0]) == 0
        return pkg._view(moe.pairs_ptr.value, (n, S, H), torch.float32).cpu().numpy().copy()
    assert launches(pkg, moe, dbank, xd, pd, wd, rows) > 1
    chunk, windows = run(0, rows), np.concatenate([run(lo, 16) for lo in range(0, rows, 16)])
    # (one flipped rounding moves a product of up to 8 times the rms by 2^-8, and with weights of up to 3.5 times theirs an element of a sum of
    # I >= 256 products by 2^-8 * 8 * 3.5 / (4 sqrt(256)) = 1.7e-3 of the largest; a lost or doubled chain by much more)
    emax, erms = rel_err(chunk, Y)
    assert emax < 4e-3 and erms < TOL, (emax, erms)
    off = [(np.linalg.norm(y - Y, axis=2) / np.linalg.norm(Y, axis=2)).mean() for y in (chunk, windows)]
    assert off[0] < 1.5 * off[1], off


@pytest.mark.parametrize("rows", [1, 16, 17, 18, 100, 128])
def test_scale_vectors_at_any_address(pkg, synth, cuda, rows):
    # the layer's calls of up to 128 rows take scale vectors that are 2-byte aligned only, on either side of the line: the bytes of
    # aligned ones
    import torch
    H, I, E, S = 512, 256, 11, 6
    dbank = synth.to_device(synth.expert_bank(91, H, I, E, svh_scale=True), cuda)
    odd = dict(dbank)
    for i, name in enumerate(n for n in dbank if n[:3] in ("suh", "svh")):
        wide = torch.zeros(dbank[name].numel() + 8, dtype=dbank[name].dtype, device=cuda)
        at = 1 + i % 3                                           # 2, 4 and 6 bytes
        odd[name] = wide[at:at + dbank[name].numel()].view_as(dbank[name]).copy_(dbank[name])
        assert odd[name].data_ptr() % 8 == 2 * at
    x, (picks, rw) = synth.activations_bf16(92, rows, H), synth.route(93, rows, E, S - 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd, pd, wd = t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw)
    moe, out = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=128)), []
    for b in (dbank, odd):
        moe.output.fill_(float("nan"))
        moe.run(b, xd, pd, wd, rows)
        torch.cuda.synchronize()
        assert int(moe.status.cpu()[0]) == 0
        out.append(moe.output[:rows].clone().view(torch.int32))
    assert torch.equal(*out)


@pytest.mark.parametrize("rows", [1, 8, 16])
@pytest.mark.parametrize("shared_rows", [(512, 1024), (3, 6), (0, 1), (5, 64), (0, 64)])
@pytest.mark.parametrize("share", [{}, dict(expert_lo=2, expert_hi=7)])
def test_shared_row_window_of_a_short_call(pkg, oracle, synth, cuda, rows, shared_rows, share):
    # a handle for large chunks whose shared expert is split by rows over the ranks, given a tail of 16 rows or fewer: none, some and
    # all of its rows are in the window
    H, I, E, S = 512, 512, 12, 4
    bank = synth.expert_bank(57, H, I, E, svh_scale=True)
    x, (picks, rw) = synth.activations_bf16(58, rows, H), synth.route(59, rows, E, S - 1)
    got = run(pkg, cuda, synth.to_device(bank, cuda), x, picks, rw, H, I, E, S, rows, synth, max_rows=64, shared_rows=shared_rows, **share)
    Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1).reshape(rows, S, H)
    lo, hi, at = share.get("expert_lo", 0), share.get("expert_hi", E), np.arange(rows)[:, None]
    here = (picks >= lo) & (picks < hi) | (picks == E) & (at >= shared_rows[0]) & (at < shared_rows[1])
    want = np.where(here[..., None], np.where((np.arange(S) == S - 1)[None, :, None], 1, rw[..., None]) * Y, 0).sum(1)
    scale = np.abs(Y).max()                              # (a share may leave a row, or all of a one-row call, without an expert)
    assert np.abs(got - want).max() < TOL * scale


@pytest.mark.parametrize("rows", [1, 5])
def test_window_without_experts_and_repeated_picks(pkg, oracle, synth, cuda, rows):
    H, I, E, S = 512, 256, 8, 4
    bank = synth.expert_bank(41, H, I, E, svh_scale=True)
    dbank = synth.to_device(bank, cuda)
    x, (picks, rw) = synth.activations_bf16(42, rows, H), synth.route(43, rows, E, S - 1)
    # nothing of the window is computed here: the partial rows are zero
    lo = next(e for e in range(E) if e not in picks)
    none = run(pkg, cuda, dbank, x, picks, rw, H, I, E, S, rows, synth, shared_exl3=0, expert_lo=lo, expert_hi=lo + 1)
    assert (none == 0).all()
    # a pick that repeats an earlier slot of its row is not computed again: with weight 0 it must not change the row
    again, rw2 = picks.copy(), rw.copy()
    again[:, 1] = again[:, 0]
    rw2[:, 1] = 0
    got = run(pkg, cuda, dbank, x, again, rw2, H, I, E, S, rows, synth)
    Y = oracle.experts_run_rows(bank, H, I, E + 1, S, x, again, mode=1)
    want = oracle.combine(Y, rw2, rows, S, H)
    assert rel_err(got, want)[0] < TOL


def test_launch_counter_wraps(pkg, oracle, synth, cuda):
    # The counter that the exchange words carry starts at 0 like the words themselves: 0 must never come round.  Rows 1..3 are first used
    # in the launch after 2^32 - 1, on words that were never written.
    import torch
    from glmflash_b200 import _view
    H, I, E, S, rows = 256, 256, 5, 3, 4
    bank = synth.expert_bank(71, H, I, E, svh_scale=True)
    dbank = synth.to_device(bank, cuda)
    x, (picks, rw) = synth.activations_bf16(72, rows, H), synth.route(73, rows, E, S - 1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xd, pd, wd = t(x.view(np.int16)).view(torch.bfloat16), t(picks), t(rw)
    moe = pkg.Moe(pkg.make_config(H, I, E, S, max_rows=rows))
    for _ in range(3):
        moe.run(dbank, xd[:1], pd[:1], wd[:1], 1)
    # the owner's allocation: status (256 bytes), the four areas of 8-byte words (one split of k each here), the counters
    up = lambda n: (n + 255) // 256 * 256
    at = 256 + sum(up(8 * rows * S * n) for n in (2 * I, H, H, I // 2)) + 384 * 4
    torch.cuda.synchronize()
    counter = _view(moe.status.data_ptr() + at, (1,), torch.int32)
    assert int(counter.cpu()[0]) == 3
    counter.fill_(-2)                                        # 2^32 - 2 launches
    want = oracle.combine(oracle.experts_run_rows(bank, H, I, E + 1, S, x, picks, mode=1), rw, rows, S, H)
    for n, epoch in ((1, -1), (rows, 2), (rows, 3), (2, 4)):
        moe.output.fill_(0)
        moe.run(dbank, xd[:n], pd[:n], wd[:n], n)
        torch.cuda.synchronize()
        assert int(moe.status.cpu()[0]) == 0 and int(counter.cpu()[0]) == epoch
        assert rel_err(moe.output[:n].cpu().numpy(), want[:n])[0] < TOL
