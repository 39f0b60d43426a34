"""Host-side decisions of the kernel library that need no device: into how many parts the many-token
product cuts its K range (the launcher's plan runs with 148 SMs when it finds no GPU)."""
import ctypes
import random
from types import SimpleNamespace

import pytest
import torch


@pytest.fixture(scope="module")
def lib():
    from pytriton_llama_b200.ops import build
    try:
        path = build.library_path()
    except build.BuildError as e:                      # no compiler on this machine
        pytest.skip(f"the kernel library cannot be built here: {e}")
    lib = ctypes.CDLL(str(path))
    lib.ptl_gemm_tc_k_parts.argtypes = [ctypes.c_int] * 3
    lib.ptl_gemm_tc_k_parts.restype = ctypes.c_int
    return lib


def test_parts_of_the_k_range(lib):
    parts = lib.ptl_gemm_tc_k_parts
    assert parts(64, 2048, 8192) == 1                  # few tokens: the other kernel path splits K over a cluster
    assert parts(2048, 2048, 8192) == 1                # 128 tiles fill the SMs
    assert parts(4096, 8192, 2048) == 1
    assert parts(300, 2048, 100) == 1                  # K no multiple of 8: not this kernel at all
    for m, n, k in [(128, 2048, 2048), (300, 2048, 8192), (1000, 1024, 1024), (65, 128, 4096)]:
        p = parts(m, n, k)
        assert 2 <= p <= 8, (m, n, k, p)
        assert -(-k // 64) // p >= 8 or p == 1, (m, n, k, p)      # at least 8 blocks of 64 values per part
    assert parts(300, 2048, 256) == 1                  # too short a K range to cut


def test_pieces_of_long_portions_fit_what_a_step_provides_for():
    """However a step's tokens are shared out, its portions beyond the walk's longest make no more portions and pieces of 64
    tokens than the launch and its workspace are laid out for, in a captured step of more token rows too; where there can be
    none, nothing is provided for."""
    from pytriton_llama_b200.ops.cuda import CudaOps
    rng = random.Random(3)
    for _ in range(2000):
        walk = rng.choice([64, 64, 1, 100])
        lens = [rng.choice([1, 1, rng.randint(1, 70), 64, 65, rng.randint(1, 700)]) for _ in range(rng.randint(1, 40))]
        rows = sum(lens) + rng.choice([0, 3, 128])
        long = [n for n in lens if n > walk]
        for exact in (True, False):
            ctx = SimpleNamespace(positions=torch.empty(sum(lens) if exact else rows), num_requests=len(lens), q_lens=lens,
                                  max_q_len=max(lens) if exact else rows, min_q_len=min(lens) if exact else 1)
            short, portions, pieces = CudaOps._portion_paths(ctx, walk)
            assert len(long) <= portions <= len(lens) and sum(-(-n // 64) for n in long) <= pieces
            assert short or len(long) == len(lens)
            assert not exact or ((portions > 0) == bool(long) and short == (len(long) < len(lens)))


def test_tiles_of_the_float32_product(lib):
    """The tile taken is close to the best of the four for row counts that divide none of them, by times measured on a B200 (us)."""
    measured = {(70, 1024): {88: 161, 84: 87, 54: 64, 44: 56}, (213, 2048): {88: 162, 84: 88, 54: 108, 44: 97},
                (150, 3072): {88: 162, 84: 87, 54: 108, 44: 97}, (129, 16384): {88: 487, 84: 399, 54: 309, 44: 335},
                (500, 2048): {88: 164, 84: 193, 54: 173, 44: 152}, (352, 8192): {88: 487, 84: 399, 54: 353, 44: 370},
                (700, 2048): {88: 257, 84: 203, 54: 180, 44: 196}, (33, 512): {88: 156, 84: 83, 54: 61, 44: 55}}
    for (M, N), us in measured.items():
        assert us[lib.ptl_gemm_simt_tile(M, N, 1)] <= 1.05 * min(us.values()), (M, N)


def test_steps_of_more_tiles_than_a_grid_holds_are_left_to_the_other_kernels(lib):
    """-2 (take another path), not an error: the kernels that these entries replaced took steps of any size."""
    p, f, i = ctypes.c_void_p(4096), ctypes.c_float(1.0), ctypes.c_int
    size = lambda *v: [i(x) for x in v]
    for n in (65536, 1 << 20):
        assert lib.ptl_chunk_attention_tc_bf16(p, *size(1024, 0), p, i(1024), None, p, p, i(4), p, *size(n, 128, 8, 2, 128, 16), f, i(256), None,
                                               None, None, i(10), f, None) == -2
        assert lib.ptl_latent_prefill_bf16(p, p, p, p, p, *size(n, 4, 8, 512, 64, 16, 10), f, i(128), None) == -2
        assert lib.ptl_latent_decode_bf16(p, None, None, p, p, p, p, p, None, *size(n, 4, 8, 512, 64, 16, 10, 1), f, None) == -2


def test_products_of_a_few_tokens_with_many_blocks_of_short_rows_are_left_to_the_other_product(lib):
    """From four tokens on: beyond four blocks of eight features an SM, three where the rows have fewer than 1,024 values; and wherever shared memory holds fewer."""
    p, i = ctypes.c_void_p(4096), ctypes.c_int
    for M, N, K in [(4, 4744, 1024), (8, 5920, 1024), (4, 3560, 768), (8, 4096, 512), (1, 5928, 512), (3, 2376, 2560)]:
        assert lib.ptl_gemm_small_bf16(p, p, p, i(M), i(N), i(K), i(N), i(0), None, None, None, i(0), None, None, i(0), i(0), ctypes.c_float(0.0), None) == -2
