"""Which kernel the tcgen05 launcher runs for a product (no GPU: the choice is made on the host), on either side of each of its lines."""
import pytest

from rllm_b200.kernels import ops, sm100

STORE, F32, ACCUM, SWIGLU, ROPE = ops.EPI_STORE, ops.EPI_STORE_F32, ops.EPI_ACCUM_F32, ops.EPI_SWIGLU, sm100.EPI_QKV_ROPE
SMS = 148


@pytest.mark.parametrize("epi,T,N,K,want", [
    # ranges of K with tiles of 64 and 128 tokens: a narrow weight of a long K
    (ACCUM, 64, 2048, 8192, (32, 8, False)), (ACCUM, 100, 2048, 8192, (64, 4, False)), (ACCUM, 128, 2048, 8192, (64, 4, False)),
    (ACCUM, 129, 2048, 8192, (128, 4, False)), (ACCUM, 256, 2048, 8192, (128, 4, False)), (ACCUM, 257, 2048, 8192, (64, 1, False)),
    (STORE, 100, 4096, 4096, (64, 2, False)), (ACCUM, 64, 4096, 4096, (64, 4, False)), (STORE, 33, 4096, 3072, (64, 4, False)),
    (ACCUM, 100, 4096, 16384, (64, 2, False)), (ACCUM, 256, 4096, 16384, (128, 2, False)), (STORE, 100, 2048, 2048, (64, 4, False)),
    # ... and not where too few SMs would have a CTA, or the ranges would not pay for their merge
    (ACCUM, 100, 4096, 4096, (64, 1, False)), (STORE, 100, 4096, 2048, (64, 1, False)), (ACCUM, 192, 4096, 10880, (64, 1, False)),
    (ACCUM, 64, 8192, 2048, (32, 2, False)), (STORE, 33, 4096, 2048, (32, 4, False)), (ACCUM, 64, 4608, 4608, (32, 4, False)),
    (ACCUM, 192, 2048, 2048, (64, 1, False)), (ACCUM, 192, 4096, 4096, (64, 1, False)), (STORE, 128, 3072, 2048, (64, 1, False)),
    (ROPE, 100, 2048, 8192, (32, 8, False)), (SWIGLU, 64, 2048, 8192, (32, 8, False)),
    # pairs of CTAs: more than 128 tokens, where the model of both kernels says so
    (SWIGLU, 128, 8192, 2048, (128, 1, False)), (SWIGLU, 129, 8192, 2048, (256, 1, True)), (SWIGLU, 2048, 8192, 2048, (256, 1, True)),
    (ACCUM, 643, 2048, 2048, (80, 1, False)), (ACCUM, 643, 2048, 8192, (80, 1, False)), (ACCUM, 1905, 2048, 8192, (224, 1, True)),
    (SWIGLU, 384, 1024, 5440, (128, 1, False)), (SWIGLU, 300, 2048, 4096, (128, 1, False)), (STORE, 1024, 4096, 1536, (256, 1, False)),
    (ACCUM, 2047, 4096, 16384, (256, 1, True)), (ACCUM, 2834, 2048, 8192, (160, 1, True)), (ROPE, 128, 3072, 2048, (64, 1, False)), (SWIGLU, 2048, 8191, 2048, (128, 1, False)),
])
def test_the_launchers_choice(epi, T, N, K, want):
    assert sm100.launch_plan(epi, T, N, K, SMS) == want


def test_no_ranges_and_no_pairs_where_they_are_not_asked_for():
    assert sm100.launch_plan(ACCUM, 128, 2048, 8192, SMS, split=False)[1] == 1
    assert sm100.launch_plan(STORE, 64, 3072, 2048, SMS, norm=True) == sm100.launch_plan(STORE, 64, 3072, 2048, SMS, split=True)
    sm100.set_pairs(-1)
    try:
        assert sm100.launch_plan(SWIGLU, 2048, 8192, 2048, SMS) == (128, 1, False)
        assert sm100.launch_plan(STORE, 2048, 3072, 2048, SMS) == (176, 1, False)
    finally:
        sm100.set_pairs(False)


def test_pairs_take_tiles_in_steps_of_32_tokens():
    """`tcgen05.mma` over two CTAs: 32 to 256 columns in steps of 32 are the shapes the kernel issues, whatever is asked for."""
    for N, K in ((2048, 2048), (3072, 2048), (2048, 8192), (4096, 16384), (6144, 4096)):
        for T in range(129, 3000, 61):
            for epi in (STORE, ACCUM, ROPE):
                tile, ranges, pairs = sm100.launch_plan(epi, T, N, K, SMS)
                assert not pairs or (tile % 32 == 0 and ranges == 1)
    try:
        for asked, width in ((176, 160), (240, 224), (80, 64), (256, 256), (33, 32)):
            sm100.set_pairs(asked)
            assert sm100.launch_plan(STORE, 1000, 2048, 2048, SMS) == (width, 1, True)
    finally:
        sm100.set_pairs(False)


def test_which_products_of_9_to_16_tokens_are_streamed_goes_with_the_gpus_sms():
    """A long K is streamed where a CTA has one job (16 features), a norm's gate/up pair where it leaves a tcgen05 tile no SM."""
    for sms in (100, 132, SMS):
        assert sm100.stream_supported(ACCUM, False, 12, 16 * sms, 8192, sm_count=sms)
        assert not sm100.stream_supported(ACCUM, False, 12, 16 * sms + 16, 8192, sm_count=sms)
        assert sm100.stream_supported(SWIGLU, True, 12, 64 * sms, 2048, sm_count=sms)
        assert not sm100.stream_supported(SWIGLU, True, 12, 64 * sms + 16, 2048, sm_count=sms)
