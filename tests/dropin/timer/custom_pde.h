// n <- old n + dt t (1 + increment / 1024), m <- n + t: whatever replays increments has to tell the
// callbacks the right time and increment.
#include <prismspf/core/pde_operator_base.h>

PRISMS_PF_BEGIN_NAMESPACE

template <unsigned int dim, unsigned int degree, typename number>
class CustomPDE : public PDEOperatorBase<dim, degree, number>
{
public:
  using ScalarValue = dealii::VectorizedArray<number>;

  CustomPDE(const UserInputParameters<dim> &_user_inputs, PhaseFieldTools<dim> &_pf_tools)
    : PDEOperatorBase<dim, degree, number>(_user_inputs, _pf_tools)
  {}

private:
  void
  set_initial_condition([[maybe_unused]] const unsigned int       &index,
                        [[maybe_unused]] const unsigned int       &component,
                        [[maybe_unused]] const dealii::Point<dim> &point,
                        [[maybe_unused]] number                   &scalar_value,
                        [[maybe_unused]] number                   &vector_component_value) const override
  {}

  void
  compute_rhs(FieldContainer<dim, degree, number> &variable_list,
              const SimulationTimer               &sim_timer,
              unsigned int                         solve_block_id) const override
  {
    const double t = sim_timer.get_time();
    if (solve_block_id == 1)
      {
        const ScalarValue n = variable_list.template get_value<Scalar, OldOne>(0);
        variable_list.set_value_term(0, n + sim_timer.get_timestep() * t * (1.0 + sim_timer.get_increment() / 1024.0));
      }
    else
      {
        const ScalarValue n = variable_list.template get_value<Scalar, Current>(0);
        variable_list.set_value_term(1, n + t);
      }
  }
};

PRISMS_PF_END_NAMESPACE
