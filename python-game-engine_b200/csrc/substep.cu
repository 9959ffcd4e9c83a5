// The operators of one substep around the pressure solve, issued from native code: the calls a
// simulator makes one by one through the operator entries, in the same order, with the same
// arguments. At 128^2 and below the GPU finished each operator before the host had issued the
// next one (128^2 float64 with Jacobi x 100: 155 us a substep, of which 75 us GPU work; 98 issued
// from here).
#include "common.cuh"

using namespace sg;

extern "C" {

int sg_substep_transport(const sg_substep* s, void* stream) {
  SG_REQUIRE(s, "null substep");
  SG_REQUIRE(s->n_emits >= 0 && (s->n_emits == 0 || s->emits), "missing emitter table");
  const int dtype = (int)s->dtype, mode = (int)s->mask_mode;
  const int64_t H = s->H, W = s->W;
  for (int64_t k = 0; k < s->n_emits; ++k) {
    const sg_emit& e = s->emits[k];
    SG_REQUIRE(e.field >= 0 && e.field <= 3, "emitter channel must be 0..3");
    if (e.field == 0)
      SG_CHECK(sg_emit_scalar(dtype, H, W, s->density, s->ld_density, e.value, s->dt, e.x, e.y, e.radius,
                              (int)e.approach, stream));
    else if (e.field == 1)
      SG_CHECK(sg_emit_scalar(dtype, H, W, s->temperature, s->ld_temperature, e.value, s->dt, e.x, e.y, e.radius,
                              (int)e.approach, stream));
    else if (e.field == 2)
      SG_CHECK(sg_emit_scalar(dtype, H, W + 1, s->u, s->ld_u, e.value, s->dt, e.x, e.y, e.radius, (int)e.approach,
                              stream));
    else
      SG_CHECK(sg_emit_scalar(dtype, H + 1, W, s->v, s->ld_v, e.value, s->dt, e.x, e.y, e.radius, (int)e.approach,
                              stream));
  }
  if (s->n_plumes > 0)
    SG_CHECK(sg_plume_sources(dtype, H, W, s->density, s->ld_density, s->u, s->ld_u, s->v, s->ld_v, (int)s->n_plumes,
                              s->plumes, s->seed, s->step, stream));
  if (s->operator_f32)
    SG_CHECK(sg_apply_forces_f32(H, W, s->v, s->ld_v, s->density, s->ld_density, s->temperature, s->ld_temperature,
                                 s->dt, s->gravity, s->buoyancy, 1.0, s->ambient, stream));
  else
    SG_CHECK(sg_apply_forces(dtype, H, W, s->v, s->ld_v, s->density, s->ld_density, s->temperature,
                             s->ld_temperature, s->dt, s->gravity, s->buoyancy, 1.0, s->ambient, 1, stream));
  const uint8_t* fmu = s->face_mask_u;
  const uint8_t* fmv = s->face_mask_v;
  if (s->advect_f32) {
    SG_CHECK(sg_advect_velocity_f32(H, W, s->u, s->ld_u, s->u_temp, s->ld_u_temp, s->v, s->ld_v, s->v_temp,
                                    s->ld_v_temp, mode, fmu, s->ld_fmu, fmv, s->ld_fmv, s->dt, s->cell_size, stream));
    SG_CHECK(sg_advect_scalar_f32(H, W, s->density, s->ld_density, s->density_temp, s->ld_density_temp, s->u_temp,
                                  s->ld_u_temp, s->v_temp, s->ld_v_temp, mode, s->is_fluid, s->ld_fluid, s->dt,
                                  s->cell_size, s->dissipation, stream));
    if (s->temperature)
      SG_CHECK(sg_advect_scalar_f32(H, W, s->temperature, s->ld_temperature, s->temperature_temp,
                                    s->ld_temperature_temp, s->u_temp, s->ld_u_temp, s->v_temp, s->ld_v_temp, mode,
                                    s->is_fluid, s->ld_fluid, s->dt, s->cell_size, 1.0, stream));
  } else {
    SG_CHECK(sg_advect_velocity(dtype, H, W, s->u, s->ld_u, s->u_temp, s->ld_u_temp, s->v, s->ld_v, s->v_temp,
                                s->ld_v_temp, mode, fmu, s->ld_fmu, fmv, s->ld_fmv, s->dt, s->cell_size, stream));
    SG_CHECK(sg_advect_scalar(dtype, H, W, s->density, s->ld_density, s->density_temp, s->ld_density_temp, s->u_temp,
                              H, W + 1, s->ld_u_temp, s->v_temp, H + 1, W, s->ld_v_temp, mode, s->is_fluid,
                              s->ld_fluid, s->dt, s->cell_size, s->dissipation, stream));
    if (s->temperature)
      SG_CHECK(sg_advect_scalar(dtype, H, W, s->temperature, s->ld_temperature, s->temperature_temp,
                                s->ld_temperature_temp, s->u_temp, H, W + 1, s->ld_u_temp, s->v_temp, H + 1, W,
                                s->ld_v_temp, mode, s->is_fluid, s->ld_fluid, s->dt, s->cell_size, 1.0, stream));
  }
  if (s->temperature)
    SG_CHECK(sg_cool_temperature(dtype, H, W, s->temperature_temp, s->ld_temperature_temp, s->ambient,
                                 s->cooling_rate, s->dt, stream));
  return sg_compute_divergence(dtype, H, W, s->u_temp, s->ld_u_temp, s->v_temp, s->ld_v_temp, s->divergence,
                               s->ld_divergence, mode, fmu, s->ld_fmu, fmv, s->ld_fmv, s->cell_size, stream);
}

int sg_substep_project(const sg_substep* s, void* stream) {
  SG_REQUIRE(s, "null substep");
  const int mode = (int)s->mask_mode, solid_mode = (int)s->solid_mode;
  // the advected velocity lies in the spare buffers; the projected one goes back to the first
  if (s->operator_f32)
    return sg_project_metrics_f32(s->H, s->W, s->u_temp, s->ld_u_temp, s->v_temp, s->ld_v_temp, s->u, s->ld_u, s->v,
                                  s->ld_v, s->pressure, s->ld_pressure, mode, s->face_mask_u, s->ld_fmu,
                                  s->face_mask_v, s->ld_fmv, s->is_fluid, s->ld_fluid, solid_mode, s->solid,
                                  s->ld_solid, s->fluid_density, s->cell_size, s->dt, s->alpha, s->reciprocal_beta,
                                  s->divergence, s->ld_divergence, s->residual, s->ld_residual, stream);
  return sg_project_metrics((int)s->dtype, s->H, s->W, s->u_temp, s->ld_u_temp, s->v_temp, s->ld_v_temp, s->u, s->ld_u,
                            s->v, s->ld_v, s->pressure, s->ld_pressure, mode, s->face_mask_u, s->ld_fmu,
                            s->face_mask_v, s->ld_fmv, s->is_fluid, s->ld_fluid, solid_mode, s->solid, s->ld_solid,
                            s->fluid_density, s->cell_size, s->dt, s->alpha, s->reciprocal_beta, s->divergence,
                            s->ld_divergence, s->residual, s->ld_residual, stream);
}

}  // extern "C"
