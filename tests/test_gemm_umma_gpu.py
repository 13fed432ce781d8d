"""Large-M route of the quantized GEMM (tcgen05 tensor cores, accumulator in tensor memory) against
the CPU oracle (tensor/quant.go matmul), through the C ABI. It takes over from 48 rows."""
import numpy as np
import pytest

from oracle import pyoracle as yo
from yuuka_b200 import cuda, synth

from .test_gemm_gpu import run_gemm, stats

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = cuda.Device(0)
    yield d
    d.close()


@pytest.mark.parametrize("dtype", [synth.Q8_0, synth.Q4_K, synth.Q6_K, synth.Q5_K])
@pytest.mark.parametrize("rows", [48, 64, 100, 256, 272, 300, 512, 600])
def test_umma_route_matches_oracle(dev, dtype, rows):
    n_out, n_in = 520, 512   # five blocks of 128 weight rows, the last one partial; two superblocks
    w = synth.normal_quant(n_out, n_in, dtype, 0.02, 300 + dtype)
    x = synth.normal_f32(rows * n_in, 1.0, 40 + rows).reshape(rows, n_in)
    want = yo.matmul(w, dtype, n_out, n_in, x)
    got = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA)
    err, cos = stats(got, want)
    # fp16 operands, fp32 accumulate; outputs have std ~0.45 at 512 columns
    assert err <= 4e-3 and cos >= 0.999999, (err, cos)


@pytest.mark.parametrize("n_out,n_in,dtype,rows", [
    (9216, 2560, synth.Q4_K, 160), (2560, 9216, synth.Q6_K, 160), (18432, 2560, synth.Q4_K, 512), (4096, 256, synth.Q8_0, 64),
])
def test_umma_route_model_shapes_and_determinism(dev, n_out, n_in, dtype, rows):
    w = synth.normal_quant(n_out, n_in, dtype, 0.02, n_out + n_in)
    x = synth.normal_f32(rows * n_in, 1.0, 4).reshape(rows, n_in)
    want = yo.matmul(w, dtype, n_out, n_in, x)
    got = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA)
    err, cos = stats(got, want)
    assert err <= 1e-2 and cos >= 0.999999, (err, cos)
    again = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA)
    assert np.array_equal(got, again)


def test_umma_route_accumulates(dev):
    n_out, n_in, rows, dtype = 640, 768, 80, synth.Q4_K
    w = synth.normal_quant(n_out, n_in, dtype, 0.02, 9)
    x = synth.normal_f32(rows * n_in, 1.0, 10).reshape(rows, n_in)
    base = synth.normal_f32(rows * n_out, 1.0, 11).reshape(rows, n_out)
    want = base + yo.matmul(w, dtype, n_out, n_in, x)
    got = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA, accumulate=base)
    err, cos = stats(got, want)
    assert err <= 4e-3 and cos >= 0.999999, (err, cos)


@pytest.mark.parametrize("n_out,n_in,rows", [
    (128, 256, 48),      # one CTA of the pair has no rows of its own; one superblock
    (257, 512, 255), (257, 512, 257),   # a row beyond the first pair; a tile one short of full and one row over
    (1001, 1536, 97),    # both halves of K on one pair of CTAs, an odd count of rows and of outputs
    (1000, 2560, 289),   # K split, two tiles of rows
    (2560, 768, 513),
    (96000, 256, 48),    # more tiles per pair than there are accumulators
    (9216, 1024, 577),   # the two halves of K in accumulators that a tile before has used
])
@pytest.mark.parametrize("dtype", [synth.Q4_K, synth.Q6_K])
def test_umma_route_at_the_edges_of_its_tiles(dev, n_out, n_in, rows, dtype):
    w = synth.normal_quant(n_out, n_in, dtype, 0.02, 5 + n_out)
    x = synth.normal_f32(rows * n_in, 1.0, rows).reshape(rows, n_in)
    want = yo.matmul(w, dtype, n_out, n_in, x)
    got = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA)
    err, cos = stats(got, want)
    assert err <= 6e-3 and cos >= 0.999999, (err, cos)


@pytest.mark.parametrize("rows", [48, 96])
@pytest.mark.parametrize("add", [False, True])
def test_umma_route_sums_parts_of_rows_that_16_byte_stores_do_not_divide(dev, rows, add):
    """1001 outputs and up to 96 rows: three parts of K, summed one value at a time."""
    n_out, n_in, dtype = 1001, 1536, synth.Q4_K
    w = synth.normal_quant(n_out, n_in, dtype, 0.02, 12)
    x = synth.normal_f32(rows * n_in, 1.0, 13).reshape(rows, n_in)
    base = synth.normal_f32(rows * n_out, 1.0, 14).reshape(rows, n_out)
    want = yo.matmul(w, dtype, n_out, n_in, x) + (base if add else 0.0)
    got = run_gemm(dev, w, dtype, n_out, n_in, x, cuda.PATH_MMA, accumulate=base if add else None)
    err, cos = stats(got, want)
    assert err <= 6e-3 and cos >= 0.999999, (err, cos)


MANY, ALWAYS = [synth.Q5_K, synth.Q8_0], [synth.Q4_K, synth.Q6_K]  # superblocks per pair that tensor memory takes


@pytest.mark.parametrize("n_out,n_in,shared_rows,rows,dtypes", [
    # parts of K on pairs of their own: tiles of 256 rows, and of 32 and 64
    (520, 2560, 900, (48, 128, 193), ALWAYS),
    # the same with enough superblocks per pair for all types: one tile of 256, three of 96 and 128
    (1100, 16384, 250, (257, 320), ALWAYS + MANY),
    # both halves of K on one pair, a last block of weight rows that is not full: two tiles of 224, and of 32 to 160 (four,
    # three and two accumulators)
    (9220, 4096, 448, (48, 97, 160, 193, 320), ALWAYS + MANY),
    # K in one piece, several tiles per pair: 256 rows, and 64 to 192 (Q8_0 only of 64 and 160, where six stages fit)
    (19200, 3072, 250, (48, 65, 128, 160, 192), ALWAYS + MANY),
    (19200, 512, 250, (48, 97, 192), ALWAYS),
    # few superblocks per pair: Q5_K and Q8_0 stay in shared memory
    (19200, 512, 250, (48, 192), MANY),
])
def test_weights_in_tensor_memory_and_in_shared_memory_give_the_same_bits(dev, n_out, n_in, shared_rows, rows, dtypes):
    """Up to 192 rows per tile the decoded weights lie in tensor memory (Q5_K and Q8_0 where a pair walks many superblocks), above in
    shared memory: the operands are the same numbers, so a row's result does not change with the rows that travel with it. (The
    tilings named are those of 148 SMs.)"""
    for dtype in dtypes:
        w = synth.normal_quant(n_out, n_in, dtype, 0.02, 700 + dtype)
        x = synth.normal_f32(shared_rows * n_in, 1.0, 31).reshape(shared_rows, n_in)
        x = np.concatenate([x, x])
        shared = run_gemm(dev, w, dtype, n_out, n_in, x[:shared_rows], cuda.PATH_MMA)
        want = yo.matmul(w, dtype, n_out, n_in, x[:8])
        # A weight s q - m rounds s, m, s q and the result to fp16, x once: each 2e-4 (rms) of a number whose deviation is at most 2.3
        # times the weight's (m is near two of them), five together at most 1e-3 of an output's deviation, 0.02 sqrt(n_in). The
        # largest of 1.5e5 such errors is 4.5 times that; twice as much is allowed.
        assert np.max(np.abs(shared[:8] - want)) <= 9e-3 * 0.02 * n_in ** 0.5
        for m in rows:
            got = run_gemm(dev, w, dtype, n_out, n_in, x[:m], cuda.PATH_MMA)
            same = min(m, shared_rows)
            assert np.array_equal(got[:same], shared[:same]), (dtype, m, float(np.abs(got[:same] - shared[:same]).max()))
            assert np.array_equal(got[same:], shared[:m - same]), (dtype, m)
