"""Which tiles of a product are divided: host rules, checked without a GPU."""
import pytest

from odc_b200 import _ext

SMS = 148


def _plan(M, N, K):
    return _ext.load().gemm_plan(M, N, K, SMS)


@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (24, 512, 512), (255, 2048, 8192), (765, 1536, 17920), (2304, 2304, 4096),
                                   (3072, 2048, 8200), (5000, 1800, 8192), (16384, 2048, 8192), (30000, 4096, 14336)])
def test_the_plan_covers_every_tile_and_its_scratch(M, N, K):
    tiles, whole, parts, scratch = _plan(M, N, K)
    assert tiles == -(-M // 256) * -(-N // 256) and 0 <= whole <= tiles
    assert (whole == tiles) == (parts == 1) == (scratch == 0)
    assert scratch == (tiles - whole) * parts * 256 * 256 * 4 and parts <= min(8, -(-K // 64))
    if parts > 1 and whole:                # whole rounds of all pairs stay as they are
        assert whole % (SMS // 2) == 0


def test_full_rounds_and_short_reductions_are_not_divided():
    assert _plan(74 * 256, 256, 8192)[2] == 1        # one tile for every pair
    tiles, whole, parts, _ = _plan(2304, 2304, 4096)   # 7 tiles more than pairs
    assert (tiles, whole) == (81, 74) and parts > 1
    assert _plan(765, 1536, 512)[2] == 1
    assert _plan(765, 1536, 17920)[1] == 0
    assert _plan(300, 200, 4096)[2] == 1             # not a product for pairs


@pytest.mark.parametrize("n_out,k_in,tokens", [(512, 512, 1900), (768, 520, 1900), (1536, 1536, 4099), (3072, 2048, 4099),
                                               (3072, 2048, 16321), (2048, 8192, 16321), (4096, 4096, 30000)])
def test_weight_gradients_are_divided_only_where_the_link_allows_it(n_out, k_in, tokens):
    """Parts that other ranks own cost their way over the link: what is divided for one rank may be whole for several, and
    the parts, sent one after the other at 770 GB/s, never take longer than the rounds of products that dividing saves."""
    plan = lambda ranks: _ext.load().scatter_plan(n_out, k_in, tokens, ranks, SMS)
    tiles, whole, parts = plan(1)
    assert parts > 1 and whole < tiles
    for ranks in (2, 8):
        n, full, parts = plan(ranks)
        assert n == tiles
        if parts > 1:
            kb, items = -(-tokens // 64), (tiles - full) * parts
            saved = (-(-tiles // (SMS // 2)) - full // (SMS // 2)) * kb - -(-items // (SMS // 2)) * -(-kb // parts)
            link = items * 256 * 256 * 4 * (ranks - 1) / ranks / 770e9
            assert link < saved * 0.285e-6   # a k-block of a tile takes about 0.28 us


def test_small_weight_gradients_stay_whole_across_ranks():
    plan = lambda ranks: _ext.load().scatter_plan(512, 512, 765, ranks, SMS)
    assert plan(1)[2] > 1 and plan(8) == (4, 4, 1)


@pytest.mark.parametrize("T", [64, 300, 1000, 4096, 16321])
@pytest.mark.parametrize("H,F", [(512, 1536), (1536, 8960), (4096, 14336)])
def test_groups_divide_what_would_outlast_them(T, H, F):
    """No product keeps parts without k-blocks, products that overwrite fp32 stay whole, and only what is longer than the work
    of a pair is divided altogether; groups of very much work are not formed."""
    plan = lambda *g: _ext.load().gemm_group_plan(list(g), SMS)
    for acc in (False, True):
        shapes = [(T, H, 2 * F, False, False), (2 * F, H, T, True, acc), (H, F, T, True, acc)]
        kb = [-(-K // 64) for _, _, K, _, _ in shapes]
        tiles = [-(-M // 256) * -(-N // 256) for M, N, *_ in shapes]
        work = sum(k * t for k, t in zip(kb, tiles))
        parts = plan(*shapes)
        if work > 12000 * (SMS // 2):   # fp32 results
            assert parts == [0, 0, 0]
            continue
        for s, k, shape in zip(parts, kb, shapes):
            assert 1 <= s <= min(8, k) and (s == 1 or not shape[3] or acc)
        if max(kb) <= work / (SMS // 2) / 2:
            assert parts == [1, 1, 1]


@pytest.mark.parametrize("M,N,K", [(765, 1536, 17920), (1904, 1536, 151936), (4096, 1536, 151936), (3072, 2048, 16400),
                                   (2304, 2304, 16400), (4096, 4096, 28672), (16321, 2048, 16640), (1000, 392, 20000)])
def test_sums_are_as_short_in_a_group_as_in_a_launch_of_their_own(M, N, K):
    """Over more than 16384, a bf16 product keeps its own parts whatever stands next to it, and so does a weight gradient that is added
    in any order."""
    ext = _ext.load()
    taken = 0
    for neighbours in ([], [(N, 512, max(M, 64), True, True)], [(4096, 512, 300, False, False), (512, 2048, 300, False, False)]):
        products = [(M, N, K, False, False)] + neighbours
        got = ext.gemm_group_tiles(products, SMS)
        if 0 in ext.gemm_group_plan(products, SMS):   # much work in bf16
            continue
        taken += 1
        assert got[0][1:] == _plan(M, N, K)[1:3] or (_plan(M, N, K)[2] == 1 and got[0][2] == 1)
        if neighbours and neighbours[0][3] and M > 16384:
            tiles, whole, parts = ext.scatter_plan(N, 512, max(M, 64), 1, SMS)
            assert got[1][2] == parts and (parts == 1 or got[1] == (tiles, whole, parts))
    assert taken


def test_groups_are_not_formed_of_many_items():
    """Products in bf16 with many rounds of items go one by one, the sooner the fewer the tokens; fp32 ones are taken together."""
    plan = lambda T, H, F, f32: _ext.load().gemm_group_plan([(T, H, 2 * F, False, False), (2 * F, H, T, f32, f32), (H, F, T, f32, f32)], SMS)
    for T, H, F, taken in ((64, 5120, 13824, False), (256, 4096, 14336, False), (512, 4096, 14336, False), (768, 4096, 14336, True), (2000, 5120, 13824, False),
                           (64, 2048, 8192, True), (256, 1536, 8960, True)):
        assert (plan(T, H, F, False) != [0, 0, 0]) == taken, (T, H, F)
        assert plan(T, H, F, True) != [0, 0, 0]
    head = lambda T, f32: _ext.load().gemm_group_plan([(T, 2048, 128256, False, False), (128256, 2048, T, f32, f32)], SMS)
    for T in (300, 1500):
        assert head(T, False) == [0, 0] != head(T, True)
    assert _ext.load().gemm_group_plan([(128256, 2048, 300, False, False)], SMS) != [0]   # nothing else gives it its factor


def test_groups_halve_the_tiles_of_what_would_outlast_them():
    columns = lambda *g: _ext.load().gemm_group_columns(list(g), SMS)
    assert columns((300, 1536, 2048, False, False), (2048, 1536, 300, False, False)) == [128, 256]
    assert columns((16321, 2048, 3072, False, False), (3072, 2048, 16321, True, True)) == [256, 256]
    assert columns((1000, 1536, 2048, False, False), (2048, 1536, 1000, False, False)) == [256, 256]   # a second round of items


def test_statistics_in_the_product_where_they_pay():
    plan = lambda rows, words, width, gradient: _ext.load().head_plan(rows, words, width, gradient, SMS)
    for gradient in (False, True):
        for rows, words, width in ((4096, 128256, 2048), (300, 151936, 1536), (4096, 4096, 512), (2000, 1024, 512), (300, 32000, 2048)):
            assert plan(rows, words, width, gradient), (rows, words, width)
        for rows, words, width in ((255, 128256, 2048), (256, 4096, 512), (300, 8192, 2048), (1200, 1024, 4096), (4096, 200, 512)):
            assert not plan(rows, words, width, gradient), (rows, words, width)
    assert plan(4096, 128256, 512, False) and not plan(4096, 128256, 512, True)


@pytest.mark.parametrize("sharded", [False, True])
@pytest.mark.parametrize("words,width", [(128256, 2048), (128256, 4096), (152064, 5120), (4096, 512), (32000, 4096), (1000, 200), (1001, 256)])
def test_the_loss_keeps_what_its_products_are_going_to_read(words, width, sharded):
    """The logits' gradient waits for the backward only where the launch that is to read it will be taken, alone or with the input
    gradient; where it is not, the fp32 matrix would be formed next to it."""
    ext, kept = _ext.load(), []
    for tokens in (1, 64, 300, 1000, 1600, 2400, 3300, 3600, 4096, 5000):
        products = [(words, width, tokens, sharded, False)] + ([(tokens, width, words, False, False)] if sharded else [])
        taken = 0 not in ext.gemm_group_plan(products, SMS) and words % 8 == 0
        fits = tokens <= 4096 and (tokens * words * 2 <= words * width * 4 or tokens * words * 2 <= 128 << 20)
        kept.append(ext.logit_grads_pay(tokens, words, width, 4096, sharded, SMS))
        assert kept[-1] == (taken and fits), tokens
    assert (True in kept) == (words % 8 == 0 and width >= 256) and not kept[-1]


def test_the_loss_forms_the_weight_gradient_at_once_where_its_product_is_refused():
    pays = lambda *a: _ext.load().logit_grads_pay(*a, 4096, sharded, SMS)
    for sharded, first, last in ((False, (1600, 128256, 2048), (3300, 128256, 2048)), (False, (800, 152064, 5120), (1200, 152064, 5120)),
                                 (True, (3300, 128256, 4096), (3600, 128256, 4096)), (True, (2200, 152064, 5120), (2500, 152064, 5120))):
        assert pays(*first) and not pays(*last)
