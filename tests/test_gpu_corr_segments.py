"""The correlation's segments (ab_corr.cu), which run over block boundaries and differ
per class of templates: a whole search gives the threshold crossings that searches of single
blocks give, each cut into segments from its own first column.  Both are sums of the
same products in FP32; a crossing may be missing from one side only within 1e-5 of its
power cut, and powers agree to 1e-5 (measured differences stay below 2e-6)."""
import numpy as np
import pytest

from presto_b200 import synth

pytestmark = pytest.mark.gpu
DT = 64e-6


def _hits(ctx, obs, fft, first=0, count=-1):
    ctx.search(obs, fft, first_block=first, max_blocks=count)
    blk, st, wi, zi, ri, pw = ctx.last_hits()
    return {tuple(k): p for k, p in zip(zip(blk, st, wi, zi, ri), pw)}


def _same(one, whole, obs, block):
    want = {k: p for k, p in whole.items() if k[0] == block}
    for k in set(one) ^ set(want):
        cut = obs.powcut[k[1]]
        assert abs((one.get(k) or want.get(k)) - cut) <= 1e-5 * cut, (k, cut)
    for k in set(one) & set(want):
        assert abs(one[k] - want[k]) <= 1e-5 * want[k], (k, one[k], want[k])
    return len(want)


@pytest.mark.parametrize("N,zmax,wmax,numharm,kw", [
    (1 << 18, 0, 0, 32, {}),                    # one template a bank; 46 blocks to a segment of the narrowest
    (1 << 18, 50, 0, 32, {}),
    (1 << 19, 690, 0, 8, {}),                   # wide templates, segments of 468 columns
    (1 << 19, 730, 0, 8, {}),                   # the widest accepted (half width 417), of 380
    (1 << 18, 730, 0, 1, dict(locpow=True)),
    (300000, 200, 0, 16, {}),
    (1 << 18, 100, 200, 16, {}),                # a bank whose reference transform wraps
    (1 << 18, 60, 100, 8, dict(locpow=True)),   # every block's own data
    (1 << 18, 60, 0, 4, dict(photon=0.7)),
    (1 << 18, 100, None, 8, {}),                # the in-memory plane, its pre-pass blocks among them
    (1 << 17, 20, None, 4, dict(rlo=700.5)),
])
def test_whole_search_is_its_blocks(ctx, ablib, N, zmax, wmax, numharm, kw):
    T = N * DT
    ps = [dict(r=0.013 * N, z=0.3 * zmax, harms=[(0.09, 0.3)] * 6), dict(r=3.1 * T, z=-0.1 * zmax, harms=[(0.07, 1.0)] * 6)]
    fft = synth.spectrum(synth.time_series(N, N + zmax, ps))
    obs = ablib.obs_init(ablib.make_params(N, DT, fft.size, zmax=zmax, wmax=wmax, numharm=numharm, sigma=1.0, **kw))
    whole = _hits(ctx, obs, fft)
    nb = ablib.num_blocks(obs)
    busy = sorted({k[0] for k in whole})
    assert busy
    for block in sorted({0, nb // 2, nb - 1, *busy[:2], *busy[len(busy) // 2:len(busy) // 2 + 2], busy[-1]}):
        _same(_hits(ctx, obs, fft, block, 1), whole, obs, block)


def test_bad_bins_spoil_their_blocks_alone(ctx, ablib):
    """A bin that is not a number, an infinite one and a stretch of zeros: every cell of the blocks whose
    windows hold them crosses (as in the blocks' own transforms), and the others are those of the
    clean spectrum."""
    N = 1 << 18
    fft = synth.spectrum(synth.time_series(N, 5, [dict(r=70001.3, z=3.0, harms=[(0.12, 0.0)])]))
    obs = ablib.obs_init(ablib.make_params(N, DT, fft.size, zmax=10, wmax=0, numharm=1, sigma=1.0))
    clean = _hits(ctx, obs, fft)
    bad = fft.copy()
    bad[50000] = np.nan
    bad[52000] = complex(0.0, np.inf)
    bad[90000:92000] = 0.0
    got = _hits(ctx, obs, bad)
    hw, step, numdata = 21, obs.rstep, 1024
    spoilt = set()
    for b in range(ablib.num_blocks(obs)):
        lo = int(obs.rlo) + b * step - hw
        win = bad[max(lo, 0):lo + numdata]
        if not np.all(np.isfinite(win)) or np.median(np.abs(win)) == 0.0:
            spoilt.add(b)
    assert len(spoilt) >= 4
    cells = obs.numz * obs.corr_uselen
    for b in spoilt:
        assert sum(k[0] == b for k in got) == cells
    near = {b + d for b in spoilt for d in (-1, 0, 1)} - spoilt
    for b in range(ablib.num_blocks(obs)):
        if b in spoilt:
            continue
        one = {k: p for k, p in got.items() if k[0] == b}
        window = bad[max(int(obs.rlo) + b * step - hw, 0):int(obs.rlo) + b * step - hw + numdata]
        if b in near and np.any(window == 0.0):
            continue                                    # its own median moved
        _same(one, clean, obs, b)


@pytest.mark.parametrize("numharm", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("zmax,wmax", [(0, 0), (70, 0), (200, 0), (40, 40)])
def test_stage_sums_are_the_per_function_sums(ctx, ablib, numharm, zmax, wmax):
    """The search's sums of a block (one and two columns a thread, tiles that overhang the block) are, bit for
    bit, the planes of its harmonics added one after another by the per-function kernel."""
    N = 1 << 17
    fft = synth.spectrum(synth.time_series(N, 11 + zmax, [dict(r=9000.3, z=0.2 * zmax, harms=[(0.1, 0.0)] * 4)]))
    obs = ablib.obs_init(ablib.make_params(N, DT, fft.size, zmax=zmax, wmax=wmax, numharm=numharm))
    block = ablib.num_blocks(obs) // 2
    got = ctx.block_stage_sums(obs, fft, block)
    ctx.set_spectrum(obs, fft)
    lo = obs.rlo + block * obs.rstep
    hi = lo + obs.rstep - 0.5
    meta, fund = ctx.subharm_fderivs_vol(obs, 1, 1, lo, hi)
    np.testing.assert_array_equal(got[0], fund)
    m, stage = 2, 1
    while m <= numharm:
        for h in range(1, m, 2):
            smeta, sub = ctx.subharm_fderivs_vol(obs, m, h, lo, hi)
            fund = ctx.add_ffdotpows(obs, meta, fund, smeta, sub, m, h, lo)
        np.testing.assert_array_equal(got[stage], fund)
        m, stage = 2 * m, stage + 1


def _hit_arrays(ctx, obs, fft, first=0, count=-1):
    ctx.search(obs, fft, first_block=first, max_blocks=count)
    blk, st, wi, zi, ri, pw = (np.asarray(a) for a in ctx.last_hits())
    key = (((blk.astype(np.int64) * 8 + st) * 128 + wi) * 4096 + zi) * 65536 + ri
    order = np.argsort(key)
    return key[order], blk[order], st[order], np.asarray(pw, np.float64)[order]


LOUD = [("quiet", 1e-17), ("quiet", 1e-6), ("bright", 1e6), ("bright", 1e8), ("bright", 3e18)]
PLACES = (20011, 40000, 77777, 100500)


def _loud(what, value, pulsars, places=PLACES):
    """A spectrum with stretches that are quieter than the rest by a large factor or bins that are far brighter
    (bin 0 too: a series that was not de-reddened), and the bins that were changed."""
    fft = synth.spectrum(synth.time_series(1 << 18, 5, pulsars)).astype(np.complex64)
    changed = np.zeros(fft.size, bool)
    for a in places if what == "quiet" else (0, *places):
        b = a + (1600 if what == "quiet" else 1)
        fft[a:b] = fft[a:b] * np.float32(value) if what == "quiet" else value
        changed[a:b] = True
    return fft, changed


def _clean_blocks(obs, changed, banks):
    """The blocks none of whose windows (of any bank) holds a changed bin."""
    import presto_b200 as pb
    out = []
    for b in range(pb.num_blocks(obs)):
        for g in banks:
            lo = int((obs.rlo + b * obs.rstep) * g["harmnum"] / g["numharm"]) - g["hw"] - 2
            if np.any(changed[max(lo, 0):lo + g["fftlen_ref"] // 2 + 4]):
                break
        else:
            out.append(b)
    return out


@pytest.mark.parametrize("what,value", LOUD)
@pytest.mark.parametrize("zmax,wmax,numharm", [(0, 0, 32), (50, 0, 16), (50, 0, 1), (20, 20, 4)])
def test_loud_and_quiet_blocks_keep_to_themselves(ctx, ablib, what, value, zmax, wmax, numharm):
    """A segment over several blocks would carry loud bins' rounding, or a scale that overflows, into blocks whose
    own windows do not hold them.  The crossings of such blocks are those of a search of the block alone, whose
    windows hold nothing loud."""
    fft, changed = _loud(what, value, [dict(r=70001.3, z=3.0, harms=[(0.12, 0.0)] * 4)],
                         PLACES[:1] if numharm == 32 else PLACES)
    obs = ablib.obs_init(ablib.make_params(1 << 18, DT, fft.size, zmax=zmax, wmax=wmax, numharm=numharm, sigma=1.0))
    whole = _hit_arrays(ctx, obs, fft)
    cuts = np.array(list(obs.powcut), np.float64)
    blocks = _clean_blocks(obs, changed, ablib.bank_geometry(obs))
    assert len(blocks) > 8
    for b in blocks:
        key, blk, st, pw = _hit_arrays(ctx, obs, fft, b, 1)
        wkey, wst, wpw = (whole[i][whole[1] == b] for i in (0, 2, 3))
        # missing from one side only within 1e-5 of the cut
        for k, s, p, other in ((key, st, pw, wkey), (wkey, wst, wpw, key)):
            lone = ~np.isin(k, other)
            assert np.all(np.abs(p[lone] - cuts[s[lone]]) <= 1e-5 * cuts[s[lone]]), (b, int(lone.sum()))
        _, i, j = np.intersect1d(key, wkey, return_indices=True)
        assert np.all(np.abs(pw[i] - wpw[j]) <= 1e-5 * pw[i]), b


@pytest.mark.parametrize("what,value", LOUD)
@pytest.mark.parametrize("zmax", [0, 50, 200])
def test_loud_and_quiet_blocks_in_the_plane(ctx, ablib, what, value, zmax):
    """The same for the in-memory plane: the rows of such a block are those of the standard mode's block alone."""
    fft, changed = _loud(what, value, [])
    kw = dict(zmax=zmax, numharm=1)
    obs = ablib.obs_init(ablib.make_params(1 << 18, DT, fft.size, wmax=None, **kw))
    std = ablib.obs_init(ablib.make_params(1 << 18, DT, fft.size, wmax=0, **kw))
    assert obs.inmem and not std.inmem
    clean = _clean_blocks(std, changed, ablib.bank_geometry(std))
    near = [b for b in clean if {b - 2, b - 1, b + 1, b + 2} - set(clean)]
    assert len(near) > 8
    for b in near:
        got, want = ctx.block_stage_sums(obs, fft, b)[0], ctx.block_stage_sums(std, fft, b)[0]
        assert np.all(np.abs(got - want) <= 1e-5 * (want + 1.0)), b


def test_plane_of_more_than_2e31_columns(ctx, ablib):
    """A forced in-memory search of more than 2^30 bins: columns past 2^31.  A line there and one at half its
    frequency: the stage-0 power is the standard mode's, the stage-1 power the sum of the two lines' (powers of
    single bins, FP32 roundings)."""
    import torch

    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    numbins, line = (1 << 30) + (1 << 15), (1 << 30) + 20000
    fft = torch.empty(numbins, dtype=torch.complex64, device="cuda")
    torch.view_as_real(fft).normal_(0.0, 0.5 ** 0.5, generator=torch.Generator(device="cuda").manual_seed(3))
    fft[line], fft[line // 2] = 30.0, 20.0
    torch.cuda.synchronize()
    kw = dict(zmax=0, numharm=2, sigma=10.0, rlo=1.0, rhi=float(numbins - 1))
    own = ablib.Context(0)
    try:
        got = {}
        for name, more in (("plane", dict(inmem=True)), ("std", dict(wmax=0))):
            obs = ablib.obs_init(ablib.make_params(2 * numbins, DT, numbins, **kw, **more))
            assert obs.inmem == (name == "plane")
            for bin in (line, line // 2):
                block = int((bin - obs.rlo) // obs.rstep)
                own.search(obs, None, first_block=block, max_blocks=1, device_ptr=fft.data_ptr())
                blk, st, wi, zi, ri, pw = own.last_hits()
                col = int(2 * (bin - (obs.rlo + block * obs.rstep)))
                got[name, bin] = {int(s): float(p) for b, s, r, p in zip(blk, st, ri, pw) if b == block and r == col}
        for bin in (line, line // 2):
            assert abs(got["plane", bin][0] - got["std", bin][0]) <= 1e-5 * got["std", bin][0]
        want = got["plane", line][0] + got["plane", line // 2][0]
        assert abs(got["plane", line][1] - want) <= 1e-6 * want
    finally:
        own.close()
        del fft
        torch.cuda.empty_cache()
