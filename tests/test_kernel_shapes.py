"""The kernels at the edges of the sizes that choose a path or a split:

- activation and binning in one cluster, one cooperative grid or separate launches, at the
  particle counts where the choice changes: keys and order exact;
- P2G and G2P with a block split into 8, 4, 2 and 1 work items, cells of 0 to 23 particles
  (the staged ranks come in windows of four), and the force operator on the same blocks;
- upload and download at ragged counts (the arrays pass through a warp's shared memory);
- C after a run of n substeps, which only the last of them writes;
- the closure's training and inference kernels at the remainders of their tiles.
"""
import numpy as np
import pytest

from helpers import rel_l2
from test_binning import _order_from_positions
from test_edge_cases import _check_state, _random_particles
from test_gpu_parity import deforming

pytestmark = pytest.mark.gpu


def _blocks(side, seed, spec):
    """Particles in side^3 blocks, 95 in each on average, in cells of 0 to 23.  (The block table
    has 16 slots per 512 particles, at least 1,024: sparser blocks would fill it.)"""
    rng = np.random.default_rng(seed)
    counts = np.array([1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 23])
    cells = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 1, 3) * 8
    cells = (cells + rng.integers(0, 8, (len(cells), 12, 3))).reshape(-1, 3)
    cells = np.repeat(cells, rng.choice(counts, len(cells)), axis=0)
    p = _random_particles(len(cells), 0.0, 1.0, seed + 1)
    p.x[:] = ((cells + 16 + rng.uniform(0.02, 0.98, cells.shape)) * spec.dx).astype(np.float32)
    # velocities and C vary smoothly, as a simulation's do
    p.v[:] = 0.5 * np.sin(5 * p.x[:, [1, 2, 0]] + 1)
    return p


@pytest.mark.parametrize("n", [4096, 32768, 32769, 1 << 20, (1 << 20) + 1])
def test_activation_and_binning_at_the_launch_limits(zs, gpu, n):
    from zsmpm_b200 import scenes
    spec = scenes.small_scene(model=0, velocity=(0.6, -0.9, 0.4))
    half = 0.5 * (n / 8) ** (1 / 3) * spec.dx
    p = _random_particles(n, 0.5 - half, 0.5 + half, n % 1000)
    with zs.Scene(spec, p) as sc:
        for step in range(2):  # after the upload every particle is counted, then the movers merged
            sc.activate_blocks()
            sc.bin_particles()
            assert (sc.binning_info() >= 0) == (step > 0)
            keys, _ = sc.download_grid()
            order, bstart = sc.download_binning()
            o_order, o_bstart = _order_from_positions(sc.download().x, keys, spec.dx)
            assert np.array_equal(order, o_order) and np.array_equal(bstart, o_bstart)
            sc.p2g()
            sc.grid_update()
            sc.g2p()
        sc.status()


# blocks: 1, 216 and 729 / 1,331 / 2,744, around the counts where a split halves on 148 SMs
@pytest.mark.parametrize("model,side", [(0, 1), (1, 6), (0, 9), (1, 11), (0, 14)])
def test_work_splits_match_oracle(zs, gpu, model, side):
    from oracle import restated
    from zsmpm_b200 import scenes
    from zsmpm_b200.implicit import ImplicitMPMSystem
    import torch
    spec = scenes.small_scene(model=model, mode=0)
    p = _blocks(side, 100 + side, spec)
    _check_state(zs, spec, p, 1)
    with zs.Scene(spec, p) as sc:
        sc.activate_blocks()
        sc.bin_particles()
        keys, _ = sc.download_grid()
        st = sc.download()
        system = ImplicitMPMSystem(sc, 1e-3)
        rng = np.random.default_rng(side)
        vel = rng.normal(0, 0.5, (len(keys) * 512, 3)).astype(np.float32)
        v = torch.from_numpy(vel.reshape(-1)).to(gpu)
        f = torch.zeros_like(v)
        system.g2p2g(v, f)
        torch.cuda.synchronize()
        sc.status()
        o32 = restated.g2p2g(spec, st.x, st.F, st.plastic, keys, vel, dt=1e-3)
        o64 = restated.g2p2g(spec, st.x, st.F, st.plastic, keys, vel, dt=1e-3, precision="f64")
        # as far from the FP64 restatement as the FP32 one, within a factor of two
        assert rel_l2(f.cpu().numpy(), o64) <= max(2 * rel_l2(o32, o64), 1e-6)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 1000])
def test_upload_download_keep_every_particle(zs, gpu, n):
    from zsmpm_b200 import scenes
    spec = scenes.small_scene(model=0)
    p = _random_particles(n, 0.44, 0.56, n)
    with zs.Scene(spec, p) as sc:
        q = sc.download()
        for k in ("m", "x", "v", "C", "F"):
            assert np.array_equal(getattr(q, k), getattr(p, k)), k
        sc.run(1)  # and in upload order after the particles were sorted
        order = sc.download()
    assert np.abs(order.x - p.x).max() <= 2 * spec.dx


def test_run_leaves_the_affine_matrix_of_its_last_substep(zs, gpu):
    from zsmpm_b200 import scenes
    spec = scenes.small_scene(model=0)
    p = deforming(scenes.generate(spec), omega=(3.0, 0.0, 8.0), squeeze=5.0)  # C of order 8
    with zs.Scene(spec, p) as sc:
        sc.run(3)
        a = sc.download()
    with zs.Scene(spec, p) as sc:
        for _ in range(3):
            sc.substep()
        b = sc.download()
    # the same substeps, up to the order in which P2G's atomics add (2^-24 a term)
    assert rel_l2(a.C, b.C) < 1e-4 and rel_l2(a.v, b.v) < 1e-6


@pytest.mark.parametrize("n", [1, 31, 63, 64, 65, 127, 640, 641, 148 * 64 + 1])
def test_closure_kernels_at_tile_remainders(zs, gpu, n):
    import torch
    from oracle import mlp
    from test_closure import DP, _closure, _kappa, random_rows
    spec, c = _closure(zs, DP)
    st = c.state_arrays()
    rows = random_rows(DP, n, n, spec.material.E, spec.material.nu)
    x = torch.from_numpy(rows).to(gpu)
    y = c.targets(x)
    loss, grad = c.loss_grad(x, y)
    out = c.infer(x, path="tcgen05_split").cpu().numpy().astype(np.float64)
    c.status()
    k, xi = _kappa(spec.material), spec.material.hardening
    xn = (mlp.inputs(DP, rows, k, xi)[0] - st["in_mean"]) * st["in_inv_std"]
    yn = mlp.net_targets(DP, rows, y.cpu().numpy(), k, xi) / st["out_scale"]
    ref_loss, ref_grad = mlp.loss_and_grad(st["params"], xn, yn)
    # as the existing tests at other row counts: FP32 sums, and split-BF16 products to 16 bits
    assert abs(loss.item() - ref_loss) <= 1e-5 * ref_loss
    assert np.linalg.norm(grad.cpu().numpy() - ref_grad) <= 1e-4 * np.linalg.norm(ref_grad)
    ref = mlp.from_net(DP, rows, mlp.forward(st["params"], xn) * st["out_scale"], k, xi)
    for lo in (0, 3):
        scale = np.linalg.norm(ref[:, lo:lo + 3]) / np.sqrt(3) + 1e-30
        for col in range(lo, lo + 3):
            assert np.linalg.norm(out[:, col] - ref[:, col]) <= 3e-4 * scale
    c.close()
