"""The six stress components come in the order xx, yy, zz, xy, yz, zx, at Gauss points
and at nodes, from the elastic displacement and from the J2 state: one strain
component at a time on a distorted box, whose stress is known in closed form."""
import dataclasses

import numpy as np
import pytest

from test_gpu_element_kernels import _box

pytestmark = pytest.mark.gpu

# displacement gradients with one non-zero strain component each
GRADS = [np.diag([1.0, 0, 0]), np.diag([0, 1.0, 0]), np.diag([0, 0, 1.0]),
         np.array([[0, 1.0, 0], [0, 0, 0], [0, 0, 0]]), np.array([[0, 0, 0], [0, 0, 1.0], [0, 0, 0]]),
         np.array([[0, 0, 0], [0, 0, 0], [1.0, 0, 0]])]


@pytest.mark.parametrize("component", range(6))
@pytest.mark.parametrize("model", ["elastic", "j2"])
def test_one_component(pkg, component, model):
    p = _box(pkg, (5, 4, 3), 3, True)
    E, nu = 200e3, 0.3
    p.props[:] = E, nu
    if model == "j2":
        p = dataclasses.replace(p, mat_model_id=pkg.MAT_J2_ISO,
                                props=np.column_stack([p.props, np.full(p.n_elems, 1e9), np.full(p.n_elems, 1e3)]))
    m = pkg.FemModel.from_problem(p)
    u = 1e-3 * (p.coords @ GRADS[component].T).ravel()
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    ref = np.zeros(6)
    if component < 3:
        ref[:3] = lam * 1e-3
        ref[component] += 2 * mu * 1e-3
    else:
        ref[component] = mu * 1e-3
    if model == "j2":
        m.internal_force(u, update_state=True)
        m.commit()
    s, vm = m.stress(u)
    ns, nvm = m.stress_nodal(u)
    # gradients of distorted elements: condition of the Jacobian times rounding
    tol = 1e-11 * np.abs(ref).max()
    assert np.abs(s.reshape(-1, 6) - ref).max() <= tol and np.abs(ns.reshape(-1, 6) - ref).max() <= tol
    d = ref[:3]
    v = np.sqrt(0.5 * ((d[0] - d[1])**2 + (d[1] - d[2])**2 + (d[2] - d[0])**2) + 3 * (ref[3:]**2).sum())
    assert np.abs(vm - v).max() <= tol and np.abs(nvm - v).max() <= tol
    m.close()
