"""The tcgen05 product's rules on sizes, as the library itself answers them, without a GPU."""
import subprocess
import sys

import pytest
import torch

from infurnace_b200.kernels.build import load_library


def _without_a_device(code):
    """What ``code`` prints in a process that sees no GPU (a crash there ends that process alone)."""
    head = "import os; os.environ['CUDA_VISIBLE_DEVICES'] = ''\nfrom infurnace_b200.kernels.build import load_library\nlib = load_library('linear_tcgen05')\n"
    run = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, (run.returncode, run.stderr[-2000:])
    return run.stdout.split()


@pytest.mark.parametrize("n,o", [(513, 1024), (2048, 1024), (2048, 4096), (1900, 192)])
def test_where_no_pair_of_sms_can_run_the_parts_are_those_of_one_tile_per_cta(n, o):
    got = int(_without_a_device(f"print(lib.ifb_linear_tcgen05_fold_parts({n}, {o}, 1))")[0])
    assert got in (2 * -(-o // 128), 2 * -(-o // 256))


PLAIN, RESIDUAL, HEADS, GATED = range(4)


@pytest.mark.parametrize("kind", [PLAIN, RESIDUAL, HEADS, GATED])
def test_the_tiles_that_are_launched_keep_the_pairs_busy(kind):
    """A product runs over pairs of SMs only where its own tiles, two whole heads wide for the fused q | k | v product, keep four
    fifths of 74 pairs busy over their rounds; and a longer k never sends it back."""
    lib = load_library("linear_tcgen05")
    taken = 0
    for n in (1, 512, 513, 768, 769, 1000, 1400, 1900, 2048, 5000):
        for o in (64, 128, 1024, 1088, 2048, 3072, 4096, 5120, 12288):
            if kind == HEADS and o % 128:
                continue
            tile = 0
            for k in (64, 512, 1024, 2048, 4096, 8192, 25600):
                f = lib.ifb_linear_tcgen05_pair_tile(kind, n, o, k, 74)
                if not f:
                    continue
                taken += 1
                assert n > 512 and f in {PLAIN: (128, 256), RESIDUAL: (128, 256), HEADS: (256,), GATED: (128,)}[kind]
                tiles = -(-n // 256) * -(-o // f)
                assert 5 * tiles >= 4 * 74 * -(-tiles // 74), (n, o, k, f)
                assert tile in (0, f)
                tile = f
    assert taken
    assert lib.ifb_linear_tcgen05_pair_tile(HEADS, 1900, 1024, 25600, 74) == 0        # 64 tiles of one head, 32 of two


# Sizes on either side of the lines for the heads' epilogue (rounds, k), and others at which those lines do not hold.
@pytest.mark.parametrize("kind,n,o,k,tile", [
    (PLAIN, 2048, 1024, 1024, 128), (PLAIN, 1000, 4096, 1024, 256), (PLAIN, 2048, 4096, 1024, 256),
    (RESIDUAL, 2048, 1024, 1024, 128), (RESIDUAL, 2048, 4096, 4096, 256),
    (HEADS, 1000, 4096, 1024, 0), (HEADS, 2048, 4096, 1024, 0), (HEADS, 1000, 4096, 4096, 0), (HEADS, 2048, 4096, 2040, 0), (HEADS, 2048, 4096, 2048, 256), (HEADS, 2048, 6144, 4096, 256),
    (GATED, 600, 3072, 1024, 128), (GATED, 2048, 12288, 4096, 128)])
def test_the_heads_of_a_short_product_stay_on_one_tile_per_cta(kind, n, o, k, tile):
    assert load_library("linear_tcgen05").ifb_linear_tcgen05_pair_tile(kind, n, o, k, 74) == tile


def test_only_a_last_round_that_leaves_half_the_pairs_idle_is_halved():
    """And a product that would not run over pairs with whole tiles takes them for the halves' sake only where the kernel it would go to needs
    a round more than the whole ones: the wide tiles, or the persistent kernel for gates from a k of 1,024 on."""
    lib = load_library("linear_tcgen05")
    whole, halves, left = 0, 0, 0
    for kind in (PLAIN, RESIDUAL, HEADS, GATED):
        for n in (1, 512, 513, 768, 818, 1000, 1100, 1400, 1900, 2048, 5000):
            for o in (64, 1000, 1024, 1088, 2048, 2304, 3072, 4096, 6144, 12288):
                rest = lib.ifb_linear_tcgen05_pair_halved(kind, n, o, 1024, 74)
                assert lib.ifb_linear_tcgen05_pair_halved(kind, n, o, 511, 74) == 0
                tiles, lone = -(-n // 256) * -(-o // (128 if kind == GATED else 256)), -(-n // 128) * -(-o // 128)
                if kind in (RESIDUAL, HEADS) or n <= 512 or o % 64 or tiles <= 74 or tiles % 74 > 37:
                    assert rest == 0, (kind, n, o)
                elif lib.ifb_linear_tcgen05_pair_tile(kind, n, o, 1024, 74):
                    assert rest == tiles % 74, (kind, n, o)
                    whole += rest > 0
                elif kind == GATED:
                    assert rest == (tiles % 74 if -(-lone // 148) > tiles // 74 else 0), (kind, n, o)
                    assert lib.ifb_linear_tcgen05_pair_halved(kind, n, o, 1016, 74) == 0
                else:
                    narrow, wide = -(-lone // 296), -(-tiles // 148)
                    assert rest == (tiles % 74 if 1.15 * wide < narrow else 0), (kind, n, o)
                    assert lib.ifb_linear_tcgen05_pair_halved(kind, n, o, 512, 74) == rest
                halves, left = halves + (rest > 0), left + (rest == 0 and 0 < tiles % 74 <= 37 < tiles)
    assert whole > 5 and halves > 15 and left > 10


# Measured on both sides: 80 tiles for 74 pairs against one round of 144 or 288 tiles, and against two of 216 or 320.
@pytest.mark.parametrize("kind,n,o,k,halved", [(GATED, 1100, 2048, 4096, 0), (PLAIN, 1100, 4096, 1024, 0), (GATED, 1280, 2048, 4096, 6), (PLAIN, 1280, 4096, 1024, 6)])
def test_halves_are_not_worth_a_round_that_the_other_kernels_do_not_need(kind, n, o, k, halved):
    assert load_library("linear_tcgen05").ifb_linear_tcgen05_pair_halved(kind, n, o, k, 74) == halved


class _Norm:
    weight = None

    class spec:
        eps = 1e-6


class _Kernels:
    """Only what the folding of a norm asks for: the parts that the library's kernels write."""

    def can_fold_norm(self, n, dtype, w, epilogue="none"):
        return True

    def fold_parts(self, o, n=None, w=None):
        lib = load_library("linear_tcgen05")
        tile = lib.ifb_linear_tcgen05_pair_tile(RESIDUAL, n, o, w.shape[1], 74) if n > 512 else 0
        return -(-o // 64) if tile else 2 * -(-o // 128) if n > 64 else -(-o // 16)

    def linear_residual_norm(self, a, w, x, weight, out, partials):
        pass


@pytest.mark.parametrize("o", [64, 192, 320, 1024, 1088, 4160])
def test_the_buffer_of_partial_sums_never_grows(o):
    """Its address is part of the steps that were recorded: small steps first, then the largest."""
    from infurnace_b200.engine.runner import _Arena
    from infurnace_b200.parts.registry import fold_residual_norm

    class Context:
        max_rows = 2048
        arena = _Arena("cpu", 2048)

        def buffer(self, name, shape, dtype, rows=None):
            return self.arena.get(name, shape, dtype, rows)
    ctx, w = Context(), torch.empty((o, 64), dtype=torch.bfloat16)
    for n in (1, 8, 64, 129, 512, 513, 1500, 2047, 2048):
        x = torch.empty((n, o))
        fold_residual_norm(_Kernels(), ctx, "mixer", torch.empty((n, 64), dtype=torch.bfloat16), w, (x, _Norm()), torch.bfloat16)
        if n == 1:
            first = ctx.arena.generation
    assert ctx.arena.generation == first


def test_the_bound_of_long_requests_holds():
    """Rows of the prompts' attention grid: never fewer than the requests with more than 16 rows, never more than the requests."""
    import itertools
    from infurnace_b200.kernels.cuda import CudaKernels
    for group in (1, 2, 4, 8, 16):
        least = 16 // group + 1
        for count in (1, 2, 3, 4):
            for lens in itertools.product((1, 2, 3, 5, 8, 9, 10, 17, 18, 30), repeat=count):
                bound = CudaKernels.long_requests(sum(lens), count, group, max(lens), min(lens))
                assert sum(q >= least for q in lens) <= bound <= count, (group, lens)
                assert CudaKernels.long_requests(sum(lens), count, group, max(lens), 1) >= bound


def test_few_requests_beside_a_prompt_are_taken_as_they_come():
    """Looking a request up, or its place by the number of keys, costs every CTA a round trip: only where CTAs have to wait for an SM."""
    rows = load_library("attention_tc").ifb_attention_tc_rows
    assert [rows(16, n, 1, 148) for n in (1, 4, 9, 10, 40)] == [1, 4, 9, 1, 1]
    assert rows(56, 16, 3, 148) == 3 and rows(56, 16, 0, 148) == 16 and rows(56, 16, 16, 148) == 16 and rows(56, 2, 1, 148) == 2
    ordered = load_library("attention_mma", {"HEAD_DIM": 128}).ifb_attention_mma_ordered
    # a portion of 65 tokens leaves 132 SMs, one of 446 tokens 92
    assert not ordered(4, 16, 8, 8, 65, 148) and ordered(16, 16, 8, 2, 446, 148) and not ordered(16, 16, 8, 2, 65, 148)
    assert ordered(64, 16, 8, 1, 65, 148) and not ordered(65, 16, 8, 1, 65, 148) and not ordered(1, 16, 8, 32, 2048, 148)
    assert ordered(2, 16, 8, 1, 2048, 148) and ordered(4, 16, 8, 8, 65, 74)
