"""Adjoint Jacobian on the B200 (plain drop-in path) vs golden values and the oracle.

Golden values: CS/algorithms/tests/Test_AdjointJacobian.cpp:123-554 (param-shift
results the reference asserts with margins 1e-7 / 1e-4).  Larger random circuits
are compared with the oracle's restatement of AdjointJacobianLQubit.hpp:212-335
(and, when built, the reference itself) and with central finite differences.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = [-np.pi / 7, np.pi / 5, 2 * np.pi / 3]


@pytest.fixture(scope="module")
def capi():
    from lightning_b200 import capi as c
    return c


def Zs(*ws):
    return [(1.0, [("PauliZ", [w])]) for w in ws]


def jac(capi, n, ops, obs, tp, dtype=np.complex128, state=None):
    sv = capi.StateVector(n, dtype)
    if state is not None:
        sv.upload(np.asarray(state, dtype=dtype))
    return sv.adjoint_jacobian(ops, obs, tp, apply_operations=True)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_golden_single_ops(capi, dtype):
    tol = 1e-7 if dtype == np.complex128 else 1e-5
    for p in np.linspace(-2 * np.pi, 2 * np.pi, 7):
        assert abs(jac(capi, 1, [("RX", [0], False, [p])], [Zs(0)], [0], dtype)[0, 0] + np.sin(p)) < tol
        assert abs(jac(capi, 1, [("RY", [0], False, [p])], [[(1.0, [("PauliX", [0])])]], [0], dtype)[0, 0]
                   - np.cos(p)) < tol
    j = jac(capi, 2, [("RX", [0], False, [P[0]])], [Zs(0), Zs(1)], [0], dtype)
    assert abs(j[0, 0] + np.sin(P[0])) < tol and abs(j[1, 0]) < tol


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_golden_three_rx(capi, dtype):
    tol = 1e-7 if dtype == np.complex128 else 1e-5
    ops = [("RX", [i], False, [P[i]]) for i in range(3)]
    j = jac(capi, 3, ops, [Zs(0), Zs(1), Zs(2)], [0, 1, 2], dtype)
    assert np.allclose(np.diag(j), -np.sin(P), atol=tol)
    j = jac(capi, 3, ops, [Zs(0), Zs(1), Zs(2)], [0, 2], dtype)
    assert abs(j[0, 0] + np.sin(P[0])) < tol and abs(j[1, 1]) < tol and abs(j[2, 1] + np.sin(P[2])) < tol
    zzz = [[(1.0, [("PauliZ", [0]), ("PauliZ", [1]), ("PauliZ", [2])])]]
    j = jac(capi, 3, ops, zzz, [0, 1, 2], dtype)
    assert np.allclose(j[0], [-0.1755096592645253, 0.26478810666384334, -0.6312451595102775], atol=tol)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_golden_mixed_xxx(capi, dtype):
    tol = 1e-7 if dtype == np.complex128 else 1e-5
    names = ["RZ", "RY", "RZ", "CNOT", "CNOT", "RZ", "RY", "RZ"]
    params = [[P[0]], [P[1]], [P[2]], [], [], [P[0]], [P[1]], [P[2]]]
    wires = [[0], [0], [0], [0, 1], [1, 2], [1], [1], [1]]
    ops = [(a, w, False, p) for a, w, p in zip(names, wires, params)]
    xxx = [[(1.0, [("PauliX", [0]), ("PauliX", [1]), ("PauliX", [2])])]]
    j = jac(capi, 3, ops, xxx, list(range(6)), dtype)
    assert np.allclose(j[0], [0.0, -0.674214427, 0.275139672, 0.275139672, -0.0129093062, 0.323846156], atol=tol)


def test_golden_decomposed_rot(capi):
    expect = [[0, -9.90819496e-01, 0], [-8.18996553e-01, 1.62526544e-01, 0], [-0.203949, 0.48593716, 0],
              [0, 1, 0], [-2.03948985e-01, 4.85937177e-01, 0], [-8.18996598e-01, 1.62526487e-01, 0],
              [0, -9.90819511e-01, 0]]
    init = [1 / np.sqrt(2), -1 / np.sqrt(2)]
    for theta, e in zip(np.linspace(-2 * np.pi, 2 * np.pi, 7), expect):
        lp = [theta, theta ** 3, np.sqrt(2) * theta]
        ops = [("RZ", [0], False, [lp[0]]), ("RY", [0], False, [lp[1]]), ("RZ", [0], False, [lp[2]])]
        j = jac(capi, 1, ops, [Zs(0)], [0, 1, 2], state=init)
        assert np.allclose(j[0], e, atol=1e-4)


def test_golden_mixed_ops_obs_tp(capi):
    lp = [0.543, 0.54, 0.1, 0.5, 1.3, -2.3, 0.5, -0.5, 0.5]
    names = ["Hadamard", "RX", "CNOT", "RZ", "RY", "RZ", "RZ", "RY", "RZ", "RZ", "RY", "CNOT"]
    params = [[], [lp[0]], [], [lp[1]], [lp[2]], [lp[3]], [lp[4]], [lp[5]], [lp[6]], [lp[7]], [lp[8]], []]
    wires = [[0], [0], [0, 1], [0], [0], [0], [0], [0], [0], [0], [1], [0, 1]]
    ops = [(a, w, False, p) for a, w, p in zip(names, wires, params)]
    obs = [[(1.0, [("PauliX", [0]), ("PauliZ", [1])])]]
    j = jac(capi, 2, ops, obs, [1, 2, 3])
    assert np.allclose(j[0], [-0.71429188, 0.04998561, -0.71904837], atol=1e-7)


def test_golden_hamiltonians(capi):
    j = jac(capi, 2, [("RX", [0], False, [P[0]])], [[(0.3, [("PauliZ", [0])]), (0.7, [("PauliZ", [1])])]], [0])
    assert abs(j[0, 0] + 0.3 * np.sin(P[0])) < 1e-7
    ops = [("RX", [i], False, [P[i]]) for i in range(3)]
    ham = [[(0.47, [("PauliZ", [0])]), (0.32, [("PauliZ", [1])]), (0.96, [("PauliZ", [2])])]]
    j = jac(capi, 3, ops, ham, [0, 2])
    assert np.allclose(j[0], [-0.47 * np.sin(P[0]), -0.96 * np.sin(P[2])], atol=1e-7)


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_random_circuit_vs_oracle(capi, dtype, ref_module=None):
    import lq_oracle as O
    import ref
    rng = np.random.default_rng(17)
    n = 8
    ops = []
    for l in range(3):
        for q in range(n):
            ops.append((["RX", "RY", "RZ", "PhaseShift"][(q + l) % 4], [q], bool((q * l) % 3 == 1),
                        [float(rng.uniform(0, 2 * np.pi))]))
        for q in range(n - 1):
            ops.append(("CNOT", [q, q + 1], False, []))
        ops += [("IsingXX", [0, 5], False, [0.3]), ("IsingYY", [2, 6], True, [0.5]), ("IsingZZ", [1, 7], False, [0.2]),
                ("IsingXY", [3, 4], False, [1.3]), ("CRX", [4, 0], False, [0.9]), ("CRY", [6, 2], True, [0.4]),
                ("CRZ", [1, 3], False, [2.2]), ("ControlledPhaseShift", [5, 7], False, [0.8]),
                ("SingleExcitation", [2, 5], False, [0.6]), ("SingleExcitationMinus", [0, 1], False, [1.1]),
                ("SingleExcitationPlus", [6, 7], True, [0.35]), ("MultiRZ", [0, 3, 6], False, [0.45]),
                ("DoubleExcitation", [0, 2, 4, 6], False, [0.7]), ("DoubleExcitationMinus", [1, 3, 5, 7], False, [0.2]),
                ("DoubleExcitationPlus", [7, 5, 3, 1], True, [1.7]), ("Hadamard", [2], False, [])]
    obs = [Zs(0), [(1.0, [("PauliX", [3]), ("PauliY", [5])])],
           [(0.4, [("PauliZ", [2]), ("PauliZ", [3])]), (-1.1, [("PauliX", [7])]), (0.2, [("Hadamard", [4])])]]
    npar = sum(1 for o in ops if len(o[3]) > 0)
    tp = list(range(0, npar, 2))
    psi = O.zero_state(n)
    want = O.adjoint_jacobian(psi, ops, obs, tp, apply_operations=True)
    got = jac(capi, n, ops, obs, tp, dtype)
    tol = 1e-12 if dtype == np.complex128 else 1e-5
    assert np.abs(got - want).max() < tol
    m = ref.load()
    if m is not None and dtype == np.complex128:
        final = O.run_circuit(n, ops)
        rj = ref.adjoint_jacobian(m, final.copy(), ops, obs, tp)
        assert np.abs(got - rj).max() < 1e-12
    # matrix operations are not differentiated but must be undone exactly in the reverse sweep
    from lightning_b200.workloads import random_unitary
    ops2 = ops + [("QubitUnitary", [1, 6], False, [], random_unitary(rng, 2)), ("RY", [6], False, [0.4])]
    npar2 = npar + 1
    want2 = O.adjoint_jacobian(O.zero_state(n), ops2, obs, list(range(npar2)), apply_operations=True)
    got2 = jac(capi, n, ops2, obs, list(range(npar2)), dtype)
    assert np.abs(got2 - want2).max() < tol


def test_layered_rotations_vs_fd(capi):
    """The plain-config circuit family at 10 qubits: adjoint vs central finite differences (FP64)."""
    import lq_oracle as O
    from lightning_b200.workloads import layered_rotations
    ops, obs, tp = layered_rotations(n=6, layers=3, seed=1234)
    got = jac(capi, 6, ops, obs, tp)
    fd = O.finite_difference_jacobian(6, ops, obs, h=1e-5)
    assert np.abs(got - fd).max() < 1e-8


def test_layered_rotations_full_size_vs_reference(capi, ref_module):
    """The plain configuration at its full size: 20 qubits, 10 layers of RX RY RZ + CNOT ladder
    (790 gates), <Z0> and the 600-parameter Jacobian, complex128, against the reference's own
    AdjointJacobianC128 (AdjointJacobianLQubit.hpp:212-335) to 1e-12."""
    import ref
    from lightning_b200.workloads import layered_rotations
    ops, obs, tp = layered_rotations()
    assert len(ops) == 790 and len(tp) == 600
    sv = capi.StateVector(20, np.complex128)
    sv.apply_ops(ops)
    ez = sv.expval(obs[0])
    got = sv.adjoint_jacobian(ops, obs, tp)
    psi = ref.run_circuit(ref_module, 20, ops)
    assert abs(ez - ref.expval(ref_module, psi.copy(), obs[0])) < 1e-12
    want = ref.adjoint_jacobian(ref_module, psi, ops, obs, tp)
    assert got.shape == (1, 600)
    assert np.abs(got - want).max() < 1e-12


def test_adjoint_errors(capi):
    with pytest.raises(capi.B200Error, match="not supported using the adjoint"):
        jac(capi, 1, [("Rot", [0], False, [0.1, 0.2, 0.3])], [Zs(0)], [0])
    with pytest.raises(capi.B200Error, match="sorted"):
        jac(capi, 1, [("RX", [0], False, [0.1]), ("RY", [0], False, [0.1])], [Zs(0)], [1, 0])


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_vjp_state(capi, dtype):
    """State-return VJP (VectorJacobianProduct.hpp:60-156) vs the oracle and the reference module."""
    import lq_oracle as O
    import ref
    from lightning_b200.workloads import layered_rotations
    rng = np.random.default_rng(9)
    n = 7
    ops, _, _ = layered_rotations(n=n, layers=2, seed=4)
    ops = ops + [("CRX", [6, 1], False, [0.3]), ("SingleExcitation", [2, 5], True, [0.8]),
                 ("MultiRZ", [0, 3, 6], False, [0.2]), ("DoubleExcitationMinus", [0, 2, 4, 6], False, [0.5])]
    psi = O.run_circuit(n, ops)
    dy = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)) / 8
    npar = sum(1 for op in ops if op[3])
    tp = list(range(1, npar, 2))
    sv = capi.StateVector(n, dtype)
    sv.upload(psi.astype(dtype))
    got = sv.vjp_state(ops, dy.astype(dtype), tp)
    want = O.vjp_state(psi.astype(dtype).astype(np.complex128), ops, dy.astype(dtype).astype(np.complex128), tp)
    tol = 1e-12 if dtype == np.complex128 else 2e-5
    assert np.abs(got - want).max() < tol
    m = ref.load()
    if m is not None and dtype == np.complex128:
        assert np.abs(got - ref.vjp_state(m, psi.copy(), ops, dy, tp)).max() < 1e-12
    import lightning_b200.lightning_qubit_ops as ours
    st = psi.astype(dtype).copy()
    svo = getattr(ours, "StateVectorC" + ("64" if dtype == np.complex64 else "128"))(st)
    sfx = "C64" if dtype == np.complex64 else "C128"
    opsd = getattr(ours.algorithms, "create_ops_list" + sfx)(
        [o[0] for o in ops], [list(o[3]) for o in ops], [list(o[1]) for o in ops], [bool(o[2]) for o in ops],
        [np.zeros(0, dtype=dtype) for _ in ops])
    res = getattr(ours.algorithms, "VectorJacobianProduct" + sfx)()(svo, opsd, dy.astype(dtype), tp)
    assert np.abs(np.asarray(res) - want).max() < tol * 10


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_adjoint_fused_sweep_every_generator(capi, dtype):
    """A 13-qubit state takes the fused reverse sweep (one observable: a Hamiltonian, the VJP
    form).  Every differentiable gate kind, constant gates and matrices on 1..4 wires, a trainable
    subset with gaps and an early exit; against the oracle's AdjointJacobianLQubit restatement,
    and against the sweep made of single calls (gate by gate, generator by generator), with one
    observable and two."""
    import lq_oracle as O
    from lightning_b200.workloads import random_unitary
    rng = np.random.default_rng(1313)
    n = 13
    diff_gates = {"RX": 1, "RY": 1, "RZ": 1, "PhaseShift": 1, "CRX": 2, "CRY": 2, "CRZ": 2,
                  "ControlledPhaseShift": 2, "IsingXX": 2, "IsingYY": 2, "IsingZZ": 2, "IsingXY": 2,
                  "SingleExcitation": 2, "SingleExcitationMinus": 2, "SingleExcitationPlus": 2,
                  "DoubleExcitation": 4, "DoubleExcitationMinus": 4, "DoubleExcitationPlus": 4, "MultiRZ": 3}
    names = list(diff_gates)
    ops = [("Hadamard", [q], False, []) for q in range(n)]
    for _ in range(140):
        r = rng.random()
        if r < 0.65:
            name = names[int(rng.integers(len(names)))]
            k = diff_gates[name]
            ops.append((name, [int(w) for w in rng.choice(n, k, replace=False)], bool(rng.random() < 0.3),
                        [float(rng.uniform(0, 2 * np.pi))]))
        elif r < 0.8:
            name = ["CNOT", "CZ", "SWAP", "Toffoli"][int(rng.integers(4))]
            ops.append((name, [int(w) for w in rng.choice(n, 3 if name == "Toffoli" else 2, replace=False)],
                        False, []))
        elif r < 0.9:
            k = int(rng.integers(1, 5))
            ops.append(("QubitUnitary", [int(w) for w in rng.choice(n, k, replace=False)], False, [],
                        random_unitary(rng, k)))
        else:
            ops.append((["S", "T", "PauliY", "Hadamard"][int(rng.integers(4))], [int(rng.integers(n))], False, []))
    npar = sum(1 for op in ops if op[3])
    tp = sorted(int(x) for x in rng.choice(npar - 10, (npar - 10) // 2, replace=False))  # gaps, early exit
    ham = [[(0.7, [("PauliZ", [0]), ("PauliZ", [5])]), (-1.2, [("PauliX", [12])]), (0.4, [("PauliY", [3])])]]
    st = O.run_circuit(n, ops)
    want = O.adjoint_jacobian(st, ops, ham, tp)
    sv = capi.StateVector(n, dtype)
    sv.upload(st.astype(dtype))
    got = sv.adjoint_jacobian(ops, ham, tp)
    tol = 1e-12 if dtype == np.complex128 else 1e-5
    assert np.abs(got - want).max() < tol
    # the sweep by single calls: one kernel a gate, a generator applied to a copy, an inner product
    lam, bra, mu = (capi.StateVector(n, dtype) for _ in range(3))
    lam.upload(st.astype(dtype))
    bra.copy_from(lam)
    bra.apply_observable(ham[0])
    single, k = np.zeros(len(tp)), npar
    for op in reversed(ops):
        if op[3]:
            k -= 1
            if k in tp:
                mu.copy_from(lam)
                scale = mu.apply_generator(op[0], op[1])
                single[tp.index(k)] = -2 * scale * (-1 if op[2] else 1) * bra.inner(mu).imag
        for s in (lam, bra):
            if len(op) > 4:
                s.apply_matrix(op[4], op[1], inverse=True)
            else:
                s.apply(op[0], op[1], not op[2], op[3])
    assert np.abs(got[0] - single).max() < tol
    # two observables
    got2 = sv.adjoint_jacobian(ops, ham + [[(1.0, [("PauliZ", [7])])]], tp)
    assert np.abs(got2[0] - got[0]).max() < tol
    want2 = O.adjoint_jacobian(st, ops, [[(1.0, [("PauliZ", [7])])]], tp)
    assert np.abs(got2[1] - want2[0]).max() < tol


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 7, 8, 9, 10, 11, 12, 14])
def test_fused_narrow_states(capi, n, dtype):
    """States around and below one shared-memory tile (padded below a warp of threads): every gate
    kind that fits the width through apply_ops_fused, and the Jacobian of one and of three
    observables, against the oracle.  Tolerances: as the other fused tests, 1e-12 and 2e-5."""
    import lq_oracle as O
    from lightning_b200.workloads import random_unitary
    rng = np.random.default_rng(100 + n)
    kinds = {"RX": (1, 1), "RY": (1, 1), "RZ": (1, 1), "PhaseShift": (1, 1), "Hadamard": (1, 0), "PauliX": (1, 0),
             "CNOT": (2, 0), "CZ": (2, 0), "SWAP": (2, 0), "CRY": (2, 1), "ControlledPhaseShift": (2, 1),
             "IsingXY": (2, 1), "IsingZZ": (2, 1), "SingleExcitationPlus": (2, 1), "Toffoli": (3, 0), "CSWAP": (3, 0),
             "DoubleExcitation": (4, 1), "DoubleExcitationMinus": (4, 1)}
    names = [k for k, (w, _) in kinds.items() if w <= n]
    ops = []
    for _ in range(70):
        name = names[int(rng.integers(len(names)))]
        w, p = kinds[name]
        ops.append((name, [int(x) for x in rng.choice(n, w, replace=False)], bool(rng.random() < 0.3),
                    [float(rng.uniform(0, 2 * np.pi))] if p else []))
    for k in range(1, min(n, 3) + 1):
        ops.append(("QubitUnitary", [int(x) for x in rng.choice(n, k, replace=False)], False, [], random_unitary(rng, k)))
    ops.append(("MultiRZ", list(range(n)), False, [0.4]))
    tol = 1e-12 if dtype == np.complex128 else 2e-5
    psi = (rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n))
    psi = (psi / np.linalg.norm(psi)).astype(dtype)
    sv = capi.StateVector(n, dtype)
    sv.upload(psi)
    sv.apply_ops_fused(ops)
    assert np.abs(sv.download() - O.run_circuit(n, ops, state=psi.astype(np.complex128))).max() < tol
    npar = sum(1 for op in ops if op[3])
    tp = list(range(0, npar, 2))
    obs = [[(1.0, [("PauliZ", [0])])], [(0.5, [("PauliX", [n - 1])]), (-0.3, [("PauliZ", [n // 2])])],
           [(1.0, [("PauliY", [n - 1])])]]
    st = sv.download()
    for o in (obs[1:2], obs):
        got = sv.adjoint_jacobian(ops, o, tp)
        assert np.abs(got - O.adjoint_jacobian(st.astype(np.complex128), ops, o, tp)).max() < tol
    assert np.array_equal(sv.download(), st)


@pytest.mark.parametrize("n", [6, 12, 14])
@pytest.mark.parametrize("nobs", [1, 3])
def test_complex64_generator_products_in_fp64(capi, n, nobs):
    """The generator products of a complex64 Jacobian are formed and summed in FP64: with one step after the
    state (a gate of each kind, or a run on one wire) and bras that are sign flips and permutations of it,
    nothing is rounded to FP32, so the Jacobian is the oracle's on the same amplitudes to FP64 rounding
    (2^n products of 1e-16; FP32 products miss by 1e-9)."""
    import lq_oracle as O
    from conftest import random_state
    rng = np.random.default_rng(n)
    psi = random_state(rng, n, np.complex64)
    sv = capi.StateVector(n, np.complex64)
    sv.upload(psi)
    obs = [[(1.0, [("PauliZ", [2])])], [(1.0, [("PauliX", [n - 1]), ("PauliZ", [1])])], [(1.0, [("PauliX", [0])])]]
    for o in ([obs[:1], obs[1:2]] if nobs == 1 else [obs]):
        for q in (0, n // 2, n - 1):
            p = (q + 1) % n
            for ops in ([("RX", [q], False, [0.4])], [("RY", [q], True, [1.4])], [("RZ", [q], False, [2.4])],
                        [("PhaseShift", [q], False, [0.9])], [("CRX", [q, p], False, [0.3])],
                        [("CRY", [p, q], False, [0.8])], [("CRZ", [q, p], False, [1.1])],
                        [("ControlledPhaseShift", [p, q], False, [0.6])], [("IsingZZ", [q, p], False, [0.7])],
                        [("MultiRZ", [q, p, (p + 1) % n], False, [0.2])],
                        [("RX", [q], False, [0.4]), ("RY", [q], False, [1.0]), ("RZ", [q], False, [2.0])]):
                tp = list(range(len(ops)))
                got = sv.adjoint_jacobian(ops, o, tp)
                want = O.adjoint_jacobian(psi.astype(np.complex128), ops, o, tp)
                assert np.abs(got - want).max() < 1e-13, (q, ops)


def test_gradient_workspace_does_not_grow_with_the_parameters(capi):
    """20 000 parameters on 20 qubits: the sweep's work memory stays below 200 MB (one partial sum per step and
    CTA for all of them would take 330), and parameters from all over the list have the shift rule's values,
    with one and with two observables."""
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    pool, high = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    n, count = 20, 20000
    rng = np.random.default_rng(8)
    angles = rng.uniform(0, 2 * np.pi, count)

    def circuit(a):
        return [op for i in range(count) for op in ((("RX", "RY")[i % 2], [i % 6], False, [float(a[i])]),
                                                    ("CNOT", [i % 6, (i + 1) % 6], False, []))]
    obs = [[(1.0, [("PauliZ", [2])]), (0.5, [("PauliX", [4])])], [(1.0, [("PauliZ", [0]), ("PauliZ", [1])])]]

    def values(a):
        sv = capi.StateVector(n)
        sv.apply_ops_fused(circuit(a))
        return np.array([sv.expval(o) for o in obs])
    sv = capi.StateVector(n)
    ops = circuit(angles)
    sv.apply_ops_fused(ops)
    used_high = 8  # cudaMemPoolAttrUsedMemHigh
    for o in (obs[:1], obs):
        assert rt.cudaMemPoolSetAttribute(pool, used_high, ctypes.byref(ctypes.c_uint64(0))) == 0
        jac = sv.adjoint_jacobian(ops, o, list(range(count)))
        assert rt.cudaMemPoolGetAttribute(pool, used_high, ctypes.byref(high)) == 0
        assert 0 < high.value < 200e6
    for k in (0, 1, 63, 64, 5000, 12345, 19999):
        shift = np.zeros(count)
        shift[k] = np.pi / 2
        want = (values(angles + shift) - values(angles - shift)) / 2
        assert np.abs(jac[:, k] - want).max() < 1e-10  # 40 000 gates of about 1e-16 each way


@pytest.mark.parametrize("n,dtype", [(22, np.complex128), (24, np.complex128), (23, np.complex64), (25, np.complex64)])
def test_several_observables_on_wide_states(capi, n, dtype):
    """Three observables where their sweeps share launches (22 qubits complex128, 23 complex64) and where each has
    its own (24, 25), with more tiles than CTAs either way and a matrix that runs on its own between the
    segments, against the oracle."""
    import lq_oracle as O
    from lightning_b200.workloads import random_unitary
    rng = np.random.default_rng(n)
    ops = [("RY", [0], False, [0.7]), ("RX", [n - 1], False, [1.3]), ("CNOT", [0, n - 1], False, []),
           ("CRZ", [n // 2, 3], False, [0.9]), ("QubitUnitary", [1, 8, 12, n - 2], False, [], random_unitary(rng, 4)),
           ("RX", [5], True, [0.4]), ("RZ", [5], False, [2.1]), ("IsingXX", [2, 9], False, [0.5])]
    obs = [[(1.0, [("PauliZ", [n - 1])])], [(0.5, [("PauliX", [5])]), (-0.3, [("PauliZ", [0])])],
           [(1.0, [("PauliY", [9]), ("PauliZ", [3])])]]
    psi = np.zeros(1 << n, dtype=np.complex128)  # a product state on the wires the circuit touches
    psi.reshape((2,) * n)[(slice(None),) * 13 + (0,) * (n - 14) + (slice(None),)] = \
        (rng.normal(size=(2,) * 14) + 1j * rng.normal(size=(2,) * 14)) / 180
    sv = capi.StateVector(n, dtype)
    sv.upload(psi.astype(dtype))
    got = sv.adjoint_jacobian(ops, obs, [0, 1, 2, 3, 4, 5])
    want = O.adjoint_jacobian(psi.astype(dtype).astype(np.complex128), ops, obs, [0, 1, 2, 3, 4, 5])
    assert np.abs(got - want).max() < (1e-12 if dtype == np.complex128 else 1e-5)
    alone = sv.adjoint_jacobian(ops, obs[1:2], [0, 1, 2, 3, 4, 5])  # one bra, lambda in place
    assert np.abs(alone[0] - want[1]).max() < (1e-12 if dtype == np.complex128 else 1e-5)


def test_more_observables_than_a_grid_dimension(capi):
    """65 600 observables on three qubits: rows from both ends equal those of a call with these alone."""
    ops = [("RX", [0], False, [0.3]), ("CNOT", [0, 1], False, []), ("RY", [2], False, [0.8]), ("CRY", [2, 0], False, [0.5])]
    kinds = [[(1.0, [(p, [q])])] for p in ("PauliZ", "PauliX", "PauliY") for q in range(3)]
    sv = capi.StateVector(3)
    sv.apply_ops_fused(ops)
    count = 65600
    got = sv.adjoint_jacobian(ops, [kinds[i % 9] for i in range(count)], [0, 1, 2])
    want = sv.adjoint_jacobian(ops, kinds, [0, 1, 2])
    assert np.abs(got - want[np.arange(count) % 9]).max() < 1e-14


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("kind", ["steps", "coefficients", "gradients"])
def test_segments_cut_by_a_limit(capi, kind, dtype):
    """Lists whose bits fit one tile but whose records do not fit one segment: more steps than it takes (160), more
    coefficients (1024: three-wire matrices take 64 or 129 each), more differentiated steps (64); the state and
    the Jacobian against the oracle."""
    import lq_oracle as O
    from conftest import random_state
    from lightning_b200.workloads import random_unitary
    rng = np.random.default_rng(len(kind))
    n, ops = 9, []
    for i in range({"steps": 330, "coefficients": 40, "gradients": 200}[kind]):
        w = [int(x) for x in rng.choice(n, 3, replace=False)]
        if kind == "steps":
            ops.append((("CNOT", "CY", "CZ", "Toffoli")[i % 4], w if i % 4 == 3 else w[:2], False, []))
        elif kind == "coefficients":
            ops.append(("QubitUnitary", w, False, [], random_unitary(rng, 3)))
        else:
            ops.append((("CRX", "CRY", "CRZ", "IsingZZ")[i % 4], w[:2], bool(i % 3), [float(rng.uniform(0, 6))]))
        if i % 20 == 0:
            ops.append(("RY", [w[0]], False, [float(rng.uniform(0, 6))]))
    psi = random_state(rng, n, dtype)
    sv = capi.StateVector(n, dtype)
    sv.upload(psi)
    sv.apply_ops_fused(ops)
    want = O.run_circuit(n, ops, state=psi.astype(np.complex128))
    assert np.abs(sv.download() - want).max() < (1e-12 if dtype == np.complex128 else 2e-5)
    tp = list(range(sum(1 for op in ops if op[3])))
    for obs in ([Zs(0)], [Zs(0), [(0.5, [("PauliX", [4])]), (1.0, [("PauliY", [8])])]]):
        st = sv.download()
        got = sv.adjoint_jacobian(ops, obs, tp)
        want = O.adjoint_jacobian(st.astype(np.complex128), ops, obs, tp)
        assert np.abs(got - want).max() < (1e-12 if dtype == np.complex128 else 1e-5)
