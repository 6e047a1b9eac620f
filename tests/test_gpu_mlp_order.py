"""The order in which minibatch training visits the samples over several epochs.

With a learning rate of zero and all parameters zero the prediction stays zero,
so an epoch's loss is the mean square of the targets it visited; batches that
leave samples out make that set differ from epoch to epoch.  The expected sets
come from a C++ program that shuffles as the trainer states it: the indices in
order, std::shuffle with one std::mt19937_64 seeded once per call."""
import shutil
import subprocess

import numpy as np
import pytest

from fvs2d_gb300.mlp import MLP

pytestmark = pytest.mark.gpu

SRC = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
int main(int, char** a) {
  const long n = std::atol(a[1]), epochs = std::atol(a[2]);
  std::mt19937_64 rng(std::strtoull(a[3], nullptr, 10));
  std::vector<int> v(n);
  for (long e = 0; e < epochs; e++) {
    for (long i = 0; i < n; i++) v[i] = (int)i;
    std::shuffle(v.begin(), v.end(), rng);
    std::fwrite(v.data(), sizeof(int), n, stdout);
  }
}
"""


def orders(tmp_path, n, epochs, seed):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "order.cpp", str(tmp_path / "order")
    src.write_text(SRC)
    subprocess.run([cxx, "-O2", "-std=c++17", str(src), "-o", exe], check=True)
    out = subprocess.run([exe, str(n), str(epochs), str(seed)], check=True, capture_output=True).stdout
    return np.frombuffer(out, np.int32).reshape(epochs, n)


# one batch an epoch behind the upload of a large set; a few batches; every
# sample in the only batch (the order does not show, the second vector does)
@pytest.mark.parametrize("n,batch,epochs", [(400_000, 200_001, 5), (5_000, 1_700, 6), (300, 300, 3), (7, 4, 1)])
def test_epoch_orders(n, batch, epochs, tmp_path):
    seed = 12345 + n
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 3)).astype(np.float32)
    y = np.exp(1.5 * rng.standard_normal((n, 1))).astype(np.float32)
    used = n // batch * batch
    ref = np.array([np.mean(y[o[:used], 0].astype(np.float64) ** 2) for o in orders(tmp_path, n, epochs, seed)])
    m = MLP(3, 16, 1, 1, seed=1)
    m.set_params(np.zeros(m.num_params(), np.float32))
    got = m.train(x, y, batch=batch, epochs=epochs, lr=0.0, seed=seed)
    m.close()
    # FP32 sums of up to 6,251 warp sums of 32 squares added one by one: relative
    # error below 6,300 * 2^-24 = 3.8e-4, and a random walk of it is 5e-6
    assert np.all(np.abs(got - ref) <= 2e-5 * ref), (got, ref)
    if used < n:
        assert np.abs(ref[:, None] - ref[None, :])[~np.eye(epochs, dtype=bool)].min(initial=1.0) > 1e-4 * ref.max()
