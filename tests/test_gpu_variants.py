"""Kernel variants at the sizes where their tiles, remainders and dispatch rules can go wrong, against the CPU oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def oracle_rows(oracle, param, bin_, x):
    m = oracle.Model(param, bin_)
    return np.stack([m.run([xi])[0] for xi in x])


@pytest.mark.parametrize("cin,cout,k,stride,h,w,n", [
    (3, 5, 3, 1, 9, 7, 2),       # single-element loads of both operands, one tile
    (4, 64, 3, 2, 17, 16, 1),    # the narrowest whole pieces, chunk of 36
    (68, 66, 3, 1, 8, 8, 1),     # 612 = three chunks split over blocks, two column tiles, exactly one row tile
    (64, 62, 1, 1, 13, 5, 1),    # 65 rows: one past a tile; columns in pairs but not in fours
    (16, 64, 3, 1, 200, 200, 1), # 128-row tiles
])
def test_fp32_cuda_core_tiles(pkg, oracle, tmp_path, cin, cout, k, stride, h, w, n):
    param, bin_ = pkg.zoo.single_conv(str(tmp_path / "c"), h=h, w=w, cin=cin, cout=cout, k=k, stride=stride, pad=k // 2)
    x = np.random.default_rng(3).uniform(-1, 1, (n, cin, h, w)).astype(np.float32)
    m = pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA)
    got = m.run(x)[0]
    assert rel_l2(got, oracle_rows(oracle, param, bin_, x)) <= 2e-6
    many = m.run(np.concatenate([x] * 5))[0]  # more tiles, the chunks in one block or in several: the same bits
    assert np.array_equal(many[:n], got) and np.array_equal(many[-n:], got)


@pytest.mark.parametrize("m,k,n", [(1, 513, 1), (65, 7, 130), (3, 1001, 1537), (129, 2050, 63)])
def test_fp32_inner_product_of_odd_extents(pkg, oracle, tmp_path, m, k, n):
    param, bin_ = pkg.zoo.inner_product(str(tmp_path / "ip"), k, n)
    x = np.random.default_rng(4).uniform(-1, 1, (m, 1, 1, k)).astype(np.float32)
    want = oracle_rows(oracle, param, bin_, x)
    assert rel_l2(pkg.Model(param, bin_).run(x)[0], want) <= 1e-5
    assert rel_l2(pkg.Model(param, bin_, accuracy_mode=pkg.FP32_CUDA).run(x)[0], want) <= 2e-6
