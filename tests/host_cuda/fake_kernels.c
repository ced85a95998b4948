/* Kernel-layer calls that do nothing and succeed, whatever their arguments. */
#define LAUNCH(name) int name() { return 0; }
LAUNCH(qmk_abs2sum) LAUNCH(qmk_adjoint_1q) LAUNCH(qmk_adjoint_diagonal) LAUNCH(qmk_adjoint_group)
LAUNCH(qmk_apply_1q) LAUNCH(qmk_apply_blocked) LAUNCH(qmk_apply_controlled)
LAUNCH(qmk_apply_diagonal) LAUNCH(qmk_apply_diagonal_group) LAUNCH(qmk_apply_group)
LAUNCH(qmk_apply_group_moves) LAUNCH(qmk_apply_phase64) LAUNCH(qmk_apply_stages)
LAUNCH(qmk_apply_swap) LAUNCH(qmk_dot_re) LAUNCH(qmk_expect_small) LAUNCH(qmk_init_basis)
LAUNCH(qmk_pauli_accum) LAUNCH(qmk_pauli_accum_local) LAUNCH(qmk_pauli_expect) LAUNCH(qmk_sample)
LAUNCH(qmk_set_wait_poll_limit) LAUNCH(qmk_take_wait_timeouts) LAUNCH(qmk_workspace_init)
LAUNCH(qmk_x_expect) LAUNCH(qmk_xfield_costate) LAUNCH(qmk_z_expect) LAUNCH(qmk_zdiag_costate)
