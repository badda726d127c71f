"""Which kernel a product goes to, where that is decided by a model of its time: the choice against measured times."""
import pytest

from ember_b200.csrc import build

# (rows, columns of the matrix, epilogue: 0 stored, 1 stored in fp32, 2 added, 3 gated), {tokens: (us on single SMs, us on pairs)}, B200,
# 148 SMs, 74 pairs at once
PRODUCTS = [
    ((4096, 4096, 2), {560: (26.1, 22.7), 601: (26.5, 22.7), 640: (26.8, 22.7), 1400: (45.3, 40.4)}),
    ((2048, 6144, 2), {256: (15.8, 16.4), 560: (20.3, 19.5), 640: (20.8, 19.4), 1600: (32.8, 33.9)}),
    ((4096, 12288, 2), {830: (77.7, 72.3), 1100: (87.0, 92.8), 1152: (87.4, 93.2), 1600: (137.8, 126.4)}),
    ((12288, 2048, 3), {560: (30.2, 29.1), 640: (30.6, 29.5), 1280: (54.9, 47.5)}),
    ((24576, 4096, 3), {440: (84.5, 73.1), 560: (105.7, 99.6), 768: (115.4, 104.9), 1024: (157.2, 136.3)}),
    ((6144, 1024, 3), {1536: (18.8, 19.5), 1600: (20.3, 23.3), 1920: (23.9, 25.9), 2047: (25.4, 26.0)}),
    ((6144, 4096, 0), {601: (30.1, 29.0), 1700: (73.5, 62.9)}),
    ((4096, 2048, 0), {384: (13.0, 13.4), 1280: (22.5, 20.5)}),
    ((4096, 1024, 0), {1280: (14.7, 13.6), 1400: (14.9, 14.0)}),
    ((10240, 5120, 0), {256: (36.4, 34.7), 300: (43.1, 51.6)}),
]
# ... of the products that finish their heads
HEAD_PRODUCTS = [
    ((1536, 1024), {512: (13.4, 14.4), 1152: (12.8, 13.3), 2047: (13.1, 13.6)}),
    ((4096, 2048), {512: (19.6, 19.4), 601: (19.1, 19.4), 1152: (19.2, 25.8), 1280: (28.3, 25.9), 2047: (31.6, 29.0)}),
    ((6144, 4096), {601: (31.4, 29.7), 768: (33.0, 30.8), 1024: (52.9, 47.2), 1792: (79.0, 68.8)}),
    ((7168, 5120), {512: (39.1, 35.3), 560: (41.2, 53.6), 768: (62.5, 54.3), 1280: (74.0, 68.1), 1920: (105.3, 123.4)}),
]


@pytest.fixture(scope="module")
def lib():
    try:
        return build.load("gemm_tc")
    except (build.BuildError, OSError) as e:
        pytest.skip(f"the product's library cannot be built or loaded here: {e}")


@pytest.fixture(scope="module")
def on_pairs(lib):
    return lib.ember_gemm_tc_on_pairs


@pytest.mark.parametrize("matrix,times", PRODUCTS, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_pairs_or_single_sms(on_pairs, matrix, times):
    """The kernel chosen is at most 5 % slower than the other one (the measurements repeat within 4 %)."""
    n, k, epilogue = matrix
    for tokens, us in times.items():
        assert us[on_pairs(tokens, n, k, epilogue, 148, 74)] <= 1.05 * min(us), (matrix, tokens)


@pytest.mark.parametrize("tokens,n,k", [(255, 4096, 4096), (1024, 1023, 4096), (1024, 4096, 1016)])
def test_single_sms_below_what_was_measured(on_pairs, tokens, n, k):
    assert not on_pairs(tokens, n, k, 2, 148, 74)


@pytest.mark.parametrize("matrix,times", HEAD_PRODUCTS, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_pairs_or_single_sms_for_heads(lib, matrix, times):
    for tokens, us in times.items():
        assert us[lib.ember_gemm_tc_qkv_on_pairs(tokens, *matrix, 148, 74)] <= 1.05 * min(us), (matrix, tokens)


@pytest.mark.parametrize("tokens,n,k", [(511, 6144, 4096), (1024, 6144, 1016), (1024, 896, 4096)])
def test_single_sms_for_heads_below_what_was_measured(lib, tokens, n, k):
    assert not lib.ember_gemm_tc_qkv_on_pairs(tokens, n, k, 148, 74)


# float32 products of few tokens: tokens a block, columns: {blocks: (us with three stages, us with eight)}
FEW = [
    (4, 2048, {16: (5.7, 4.7), 56: (6.5, 5.6), 74: (6.1, 4.9), 128: (9.0, 5.9), 148: (6.3, 5.4)}),
    (8, 2048, {56: (9.0, 7.9), 128: (12.8, 8.2), 146: (12.4, 8.1), 192: (12.5, 14.5)}),
    (16, 1024, {8: (5.7, 6.4), 37: (5.6, 6.5), 64: (7.7, 6.6), 74: (5.6, 6.6), 128: (9.3, 7.0), 148: (5.7, 6.8), 192: (9.4, 11.9)}),
    (16, 2048, {8: (9.7, 10.9), 32: (9.9, 10.9), 64: (13.7, 11.1), 74: (9.7, 11.2), 147: (16.8, 11.6), 148: (9.8, 11.6), 149: (16.6, 18.9)}),
    (16, 3072, {16: (13.8, 14.9), 64: (19.7, 14.9), 148: (13.9, 15.4)}),
]


@pytest.mark.parametrize("tokens,columns,times", FEW, ids=lambda v: str(v) if isinstance(v, int) else "")
def test_how_far_products_of_few_tokens_look_ahead(tokens, columns, times):
    try:
        far = build.load("gemm_simt").ember_gemm_f32_few_looks_far
    except (build.BuildError, OSError) as e:
        pytest.skip(f"the product's library cannot be built or loaded here: {e}")
    for blocks, us in times.items():
        assert us[far(tokens, blocks)] <= 1.05 * min(us), (tokens, columns, blocks)


# float32 products of more tokens: (rows, columns of the matrix): {tokens: (us on tiles, us on clusters)}
MANY = [
    ((512, 1024), {65: (20.0, 18.9), 280: (19.9, 20.0), 520: (20.0, 27.2), 600: (37.2, 29.0), 1100: (39.1, 44.1)}),
    ((768, 1024), {340: (20.0, 27.5), 410: (37.8, 29.2), 720: (39.1, 44.6), 2048: (112.7, 98.1)}),
    ((1024, 1024), {200: (20.0, 20.0), 280: (20.0, 29.1), 300: (37.1, 29.3), 520: (39.0, 43.7), 640: (57.1, 46.2)}),
    ((1280, 1024), {200: (20.0, 27.9), 300: (38.6, 30.1), 1024: (94.5, 87.4)}),
    ((1536, 1024), {160: (20.0, 27.8), 200: (37.1, 28.9), 340: (38.9, 44.6)}),
    ((2048, 1024), {150: (37.3, 29.5), 280: (38.9, 45.9), 300: (55.8, 46.2), 1024: (133.0, 131.3)}),
    ((1280, 3072), {200: (54.0, 69.1), 300: (103.2, 71.8), 2048: (456.4, 413.4)}),
    ((64, 1024), {33: (19.4, 12.7), 640: (19.9, 14.3)}),
    ((2304, 1024), {65: (20.1, 25.8), 200: (38.9, 43.6)}),
]


@pytest.mark.parametrize("matrix,times", MANY, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "")
def test_tiles_or_clusters(matrix, times):
    try:
        clusters = build.load("gemm_simt").ember_gemm_f32_clusters
    except (build.BuildError, OSError) as e:
        pytest.skip(f"the product's library cannot be built or loaded here: {e}")
    for tokens, us in times.items():
        assert us[clusters(tokens, *matrix)] <= 1.05 * min(us), (matrix, tokens)
    n = matrix[0]
    assert not any(clusters(m, n, k) for m in (33, 64, 300, 2048) for k in (64, 256, 508))
    assert clusters(33, 64, 512) and not clusters(280, 1024, 512)
