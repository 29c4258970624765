"""The one-kernel training pass (tb_mlp_loss_grad) against the same pass made
of the single kernels, at batches around its tile of 64 samples and around
one tile per SM, with and without weights, for one to ten field sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _by_kernels(mlp, X, T, n_out, w):
    """Loss and gradients from forward(keep=True) and the tb_mlp_* kernels."""
    import torch
    from traceon_b200 import backend as B
    from traceon_b200 import surrogate as SG
    M = X.shape[0]
    out, pre, acts = mlp.forward(X, keep=True)
    g = torch.empty((M, SG.OUT), dtype=torch.bfloat16, device=X.device)
    part = torch.empty((M * SG.OUT + 255) // 256, dtype=torch.float32, device=X.device)
    SG._call('tb_mlp_mse_grad', out.data_ptr(), T.data_ptr(), B._ptr(w), g.data_ptr(), part.data_ptr(), M, SG.OUT, n_out,
             SG._s())
    grad = torch.empty_like(mlp.p)
    for li in range(len(SG.LAYERS) - 1, -1, -1):
        W, b, fin, fout = SG.LAYERS[li]
        SG._call('tb_mlp_gemm', g.data_ptr(), fout, 1, acts[li].data_ptr(), fin, 1, mlp._w(grad, W).data_ptr(), fin,
                 fout, fin, M, 0, SG._s())
        SG._call('tb_mlp_colsum', g.data_ptr(), mlp._w(grad, b).data_ptr(), M, fout, SG._s())
        if li:
            dA = torch.empty((M, fin), dtype=torch.float32, device=X.device)
            SG._call('tb_mlp_gemm', g.data_ptr(), fout, 0, mlp._w(mlp.pb, W).data_ptr(), fin, 1, dA.data_ptr(), fin, M,
                     fin, fout, 0, SG._s())
            g = torch.empty((M, fin), dtype=torch.bfloat16, device=X.device)
            SG._call('tb_mlp_silu_back', dA.data_ptr(), pre[li - 1].data_ptr(), g.data_ptr(), M * fin, SG._s())
    return float(part.double().sum()) / (M * n_out), grad


@pytest.mark.parametrize('M, n_out, weighted', [(1, 3, False), (63, 1, True), (64, 30, False), (65, 9, True),
                                                (1000, 9, True), (64 * 148, 6, False), (64 * 148 + 1, 9, True),
                                                (20011, 9, False)])
def test_loss_and_grad_equals_the_kernels(cuda, M, n_out, weighted):
    import torch
    from traceon_b200 import surrogate as SG
    rng = np.random.default_rng(M + n_out)
    mlp = SG.MLP(seed=n_out)
    for name in ('b1', 'b2', 'b3', 'b4', 'b5'):
        mlp._w(mlp.p, name).uniform_(-0.2, 0.2, generator=torch.Generator('cuda').manual_seed(M))
    X = torch.as_tensor(rng.uniform(-1, 1, (M, 16)), device='cuda').to(torch.bfloat16)
    T = torch.as_tensor(rng.standard_normal((M, n_out)), device='cuda', dtype=torch.float32)
    w = torch.as_tensor(rng.uniform(0.2, 3, M), device='cuda', dtype=torch.float32) if weighted else None
    want_loss, want = _by_kernels(mlp, X, T, n_out, w)
    loss = mlp.loss_and_grad(X, T, n_out, w)
    first = mlp.g.clone()
    # the same products of BF16 values; FP32 sums over up to 2e4 samples in another order: 2^-24 sqrt(M) of the sum
    # of magnitudes, which for random targets is sqrt(M) times the sum's own size
    tol = 2.0 ** -24 * 4 * max(M, 64) ** 0.5
    assert abs(float(loss) - want_loss) <= tol * want_loss
    for name, (o, n) in SG.OFF.items():
        a, b = first[o:o + n].double(), want[o:o + n].double()
        assert float((a - b).norm()) <= tol * float(b.norm()), name
    mlp.loss_and_grad(X, T, n_out, w)
    assert torch.equal(first, mlp.g)  # a fixed order of the sums
