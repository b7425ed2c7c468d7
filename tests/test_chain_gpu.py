"""Forward kinematics and contact flags of batched arms at the edges of the
kernels' blocks: chains of both forms, configuration counts around a block."""
import numpy as np
import pytest

from distance3d_gb300.robot import SelfCollisionBatch, SerialArm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dof", [2, 7, 30, 31])
@pytest.mark.parametrize("configs", [1, 8, 9])
def test_fk_and_contacts(dof, configs):
    arm = SerialArm.synthetic(seed=dof, dof=dof, n_bodies=13)
    if not len(arm.pair_table()):
        arm = SerialArm(arm.joint_axis, arm.joint_origin, np.where(np.arange(13) < 6, 0, dof), arm.body_origin,
                        arm.body_type, arm.body_params)
    q = np.random.default_rng(dof).uniform(-np.pi, np.pi, (configs, dof))
    b = SelfCollisionBatch(arm, configs, precision="fp64", graph=False)
    r = {k: v.cpu().numpy() for k, v in b.run(q).items()}
    want = np.stack([arm.fk(x) for x in q])
    # 2 dof transform products of a few roundings each (2^-53) on coordinates below 13 m
    assert np.max(np.abs(b.poses.cpu().numpy().reshape(want.shape) - want)) < 13 * 2 * dof * 8 * 2.0 ** -53
    hit = r["dist"] == 0.0
    flags = np.zeros((configs, arm.n_bodies), dtype=bool)
    for p, (i, j) in enumerate(arm.pair_table()):
        flags[:, i] |= hit[:, p]
        flags[:, j] |= hit[:, p]
    assert np.array_equal(r["contacts"], flags) and np.array_equal(r["any"], flags.any(axis=1))
