"""How a call is cut (fa_fwd_plan, host arithmetic): the plan goes by the keys that the masks leave visible."""
import pytest

from plan_util import B200_CLUSTERS, plan


@pytest.mark.parametrize("B,H,Hk,Nq,Nk,kw", [
    (1, 16, 16, 256, 8192, {}),              # a prompt written into a longer cache: two KV tiles are visible
    (1, 32, 8, 512, 32768, {}),
    (1, 32, 8, 300, 32768, {}),
    (1, 32, 8, 300, 8492, {}),
    (8, 32, 8, 22, 2839, {}),
    (1, 16, 16, 256, 8192, dict(k_pos0=8000, q_pos0=8000)),
    (1, 16, 16, 256, 8192, dict(causal=False, window=(-1, 0))),    # a right window alone bounds it as well
])
def test_keys_that_no_query_sees_do_not_count(B, H, Hk, Nq, Nk, kw):
    got = plan(B, H, Nq, Nk, 128, heads_k=Hk, **dict(dict(causal=True), **kw))
    assert (got.decode, got.parts, got.staged, got.stacked_rows) == (0, 1, 0, 0)


def test_the_same_blocks_at_the_end_of_the_cache_are_cut():
    assert plan(1, 16, 256, 8192, 128, causal=True, q_pos0=7936).parts > 1
    got = plan(1, 32, 300, 8492, 128, heads_k=8, causal=True, q_pos0=8192)
    assert got.parts > 1 and got.merged == 1 and got.stacked_rows == 300


@pytest.mark.parametrize("kw", [dict(causal=True), dict(causal=True, window=(300, 0)), dict(window=(100, 60))])
def test_the_plan_of_a_block_is_that_of_its_visible_keys(kw):
    # (cut off at the last visible key, the cache gives the same plan; positions on both sides of the tiles' edges)
    for q0 in (0, 127, 128, 1000, 3000):
        for Nq in (9, 128, 129, 300):
            right = kw["window"][1] if kw.get("window", (-1, -1))[1] >= 0 else 0
            whole = plan(1, 8, Nq, 9000, 64, heads_k=2, q_pos0=q0, **kw)
            short = plan(1, 8, Nq, (q0 + Nq + 255) // 128 * 128 + (right + 127) // 128 * 128, 64, heads_k=2, q_pos0=q0, **kw)
            assert bytes(whole) == bytes(short), (q0, Nq, kw)


@pytest.mark.parametrize("sms,clusters", [(148, B200_CLUSTERS), (132, (0, 132, 66, 40, 30, 24, 18, 12, 12, 12, 10, 7, 7, 7, 7, 7, 6)),
                                          (148, (0, 148) + (0,) * 15)])
@pytest.mark.parametrize("Nq,per_sm", [(256, 1), (100, 2)])
def test_the_clusters_of_a_split_are_resident_at_once(sms, clusters, Nq, per_sm):
    seen = set()
    for blocks in range(1, 200):
        for Nk in (500, 1024, 2419, 8492):
            parts = plan(1, blocks, Nq, Nk, 128, sms=sms, clusters=clusters).parts
            seen.add(parts)
            room = clusters[parts] if per_sm == 1 else max(2 * clusters[parts], clusters[(parts + 1) // 2])
            assert parts == 1 or blocks <= room, (blocks, Nk, parts)
    assert (seen == {1}) == (clusters[2] == 0)


@pytest.mark.parametrize("B,H,Hk,Nq,Nk,causal,parts", [
    (2, 32, 8, 62, 2419, True, (4, 5)),      # 16 stacked blocks: 20.7 us in four parts, 40.4 in seven, 31.7 unsplit and unstacked
    (1, 16, 16, 256, 2419, False, (4, 5)),
    (1, 48, 48, 256, 8492, False, (2,)),     # 45 clusters of three fit, not 48
    (1, 48, 48, 100, 1024, False, (1,)),     # 14.4 us unsplit, 15.7 in four parts
    (1, 32, 8, 300, 8492, True, (3,)),
    (8, 16, 16, 2048, 2048, True, (1,)),
])
def test_part_counts(B, H, Hk, Nq, Nk, causal, parts):
    assert plan(B, H, Nq, Nk, 128, heads_k=Hk, causal=causal, q_pos0=Nk - Nq if causal else 0).parts in parts


def test_decode_on_a_device_without_clusters():
    got = [plan(1, 8, Nq, Nk, 128, heads_k=2, num_splits=s, clusters=(0, 148) + (0,) * 15)
           for Nq in (1, 4, 8) for Nk in (100, 5000, 300000) for s in (0, 1)]
    assert all(p.decode and not p.merged for p in got) and any(p.parts > 16 for p in got)


@pytest.mark.parametrize("splits", [1, 3, 4, 16, 20])
def test_decode_with_dropout_keeps_the_callers_splits(splits):
    for B, H, Hk, Nq in ((1, 8, 8, 1), (2, 64, 8, 3), (16, 32, 8, 4)):
        got = plan(B, H, Nq, 5000, 128, heads_k=Hk, p_dropout=0.1, num_splits=splits)
        assert got.parts == splits and got.merged == (splits in (4, 16))
        alone = plan(B, H, Nq, 5000, 128, heads_k=Hk, p_dropout=0.1, num_splits=splits, clusters=(0, 148) + (0,) * 15)
        assert alone.parts == splits and not alone.merged  # (the combine kernel)
